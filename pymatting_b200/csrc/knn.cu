// k-nearest-neighbour matting Laplacian (knn_laplacian,
// pymatting/laplacian/knn_laplacian.py) on the device.
//
// Features per pixel: (r, g, b, dw x, dw y) in float32 with x, y the
// numpy.linspace(0, 1, .) grids, one pass per (k, dw). Neighbours come from
// an exact search with the reference k-d tree's distance
// (pymatting/util/kdtree.py:_find_knn: float32 squared differences summed in
// float64), keeping the k smallest by (distance, index); a distance that is not
// a number (a feature that is not finite) counts as infinite. The points are
// brought into the order of a 5-D Morton curve first, so that 32 consecutive
// ones (a tile) lie close together; tiles whose bounding box is farther than
// every query's k-th distance are skipped. The reference keeps the first found
// among equal distances in its tree order, so the two differ only where the
// k-th distance is tied.
//
// W = sum over passes of B + B^T (B_ij = 1, or 1 - |f_i - f_j|_1 / 5 for the
// soft kernel), assembled per row: the row's own neighbours, then the rows
// that list it. Each row is sorted by column, duplicates are summed in a
// fixed order, and the row is normalised: L = I - diag(1 / rowsum(W)) W.

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "pm_common.cuh"

int pmb_scan_exclusive(int64_t* v, int64_t n, int64_t* chunk_scratch, int64_t* total,
                       cudaStream_t s);

namespace pmb {
namespace knn {

constexpr int kMaxK = 64;
constexpr int kDims = 5;

// Order-preserving map of floats to unsigned (for atomic minima and maxima).
__device__ __forceinline__ unsigned ordered(float v) {
    const unsigned u = __float_as_uint(v);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float unordered(unsigned u) {
    return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}

__device__ __forceinline__ bool all_finite(const float (&f)[kDims]) {
    bool ok = true;
#pragma unroll
    for (int d = 0; d < kDims; ++d) ok = ok && isfinite(f[d]);
    return ok;
}

// Features, and the extent of the finite ones: ext[d] = smallest, ext[kDims + d]
// = largest (ordered; the smallest inverted, so that both start at 0 and grow).
__global__ void __launch_bounds__(256) k_features(const double* __restrict__ image, int h, int w, double dw,
                                                  float* __restrict__ f, unsigned* ext) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const bool in = i < (long long)h * w;
    float v[kDims];
    if (in) {
        const int y = (int)(i / w), x = (int)(i % w);
        // numpy.linspace(0, 1, num): j * (1 / (num - 1)), last element exactly 1
        const double sx = w > 1 ? 1.0 / (double)(w - 1) : 0.0;
        const double sy = h > 1 ? 1.0 / (double)(h - 1) : 0.0;
        const double xv = (w > 1 && x == w - 1) ? 1.0 : (double)x * sx;
        const double yv = (h > 1 && y == h - 1) ? 1.0 : (double)y * sy;
        v[0] = (float)image[i * 3 + 0];
        v[1] = (float)image[i * 3 + 1];
        v[2] = (float)image[i * 3 + 2];
        v[3] = (float)(dw * xv);
        v[4] = (float)(dw * yv);
    }
    __shared__ unsigned s_ext[2 * kDims];
    if (threadIdx.x < 2 * kDims) s_ext[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int d = 0; d < kDims; ++d) {
        const bool ok = in && isfinite(v[d]);
        const unsigned o = ok ? ordered(v[d]) : 0u;
        const unsigned hi = __reduce_max_sync(0xffffffffu, o);
        const unsigned lo = __reduce_max_sync(0xffffffffu, ok ? ~o : 0u);
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&s_ext[d], lo);
            atomicMax(&s_ext[kDims + d], hi);
        }
        if (in) f[i * kDims + d] = v[d];
    }
    __syncthreads();
    if (threadIdx.x < 2 * kDims) atomicMax(&ext[threadIdx.x], s_ext[threadIdx.x]);
}

constexpr int kTile = 32;
constexpr int kCellBits = 4;                              // of every dimension
constexpr int kCells = 1 << (kCellBits * kDims);          // 2^20 buckets

// Morton code of the cell that holds a point. Cells are cubes: 2^BITS of them
// along the widest dimension.
template <int BITS>
__device__ __forceinline__ int cell_of(const float (&f)[kDims], const unsigned* ext) {
    float lo[kDims], widest = 0.f;
#pragma unroll
    for (int d = 0; d < kDims; ++d) {
        lo[d] = unordered(~ext[d]);
        widest = fmaxf(widest, unordered(ext[kDims + d]) - lo[d]);
    }
    const float inv = widest > 0.f ? (float)(1 << BITS) / widest : 0.f;
    int code = 0;
#pragma unroll
    for (int d = 0; d < kDims; ++d) {
        const int c = min(max((int)((f[d] - lo[d]) * inv), 0), (1 << BITS) - 1);
#pragma unroll
        for (int b = 0; b < BITS; ++b) code |= ((c >> b) & 1) << (b * kDims + d);
    }
    return code;
}

__global__ void k_cell_count(const float* __restrict__ f, long long n, const unsigned* __restrict__ ext,
                             int* __restrict__ cell, int64_t* hist) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float v[kDims];
#pragma unroll
    for (int d = 0; d < kDims; ++d) v[d] = f[i * kDims + d];
    const int c = cell_of<kCellBits>(v, ext);
    cell[i] = c;
    atomicAdd((unsigned long long*)(hist + c), 1ull);
}

// Points in cell order: sf[d * np + pos], index in sidx[pos]. The order within
// a cell is arbitrary, which changes neither the boxes' validity nor the k
// smallest by (distance, index).
__global__ void k_reorder(const float* __restrict__ f, long long n, long long np, const int* __restrict__ cell,
                          int64_t* next, float* __restrict__ sf, int* __restrict__ sidx) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long pos = (long long)atomicAdd((unsigned long long*)(next + cell[i]), 1ull);
#pragma unroll
    for (int d = 0; d < kDims; ++d) sf[d * np + pos] = f[i * kDims + d];
    sidx[pos] = (int)i;
}

// The buckets' cells are wide for a tile of 32 points where many points share
// one: windows of kWindow points are sorted by a finer code (kFineBits a
// dimension), which keeps the order of the buckets inside a window.
constexpr int kWindow = 1024, kFineBits = 6;

__global__ void __launch_bounds__(kWindow / 2) k_refine(long long n, long long np, const unsigned* __restrict__ ext,
                                                        float* __restrict__ sf, int* __restrict__ sidx) {
    __shared__ unsigned long long key[kWindow];
    __shared__ float col[kWindow];
    const long long p0 = blockIdx.x * (long long)kWindow;
    const int m = (int)min((long long)kWindow, n - p0), tid = threadIdx.x;
    for (int e = tid; e < kWindow; e += kWindow / 2) {
        unsigned long long v = ~0ull;
        if (e < m) {
            float f[kDims];
#pragma unroll
            for (int d = 0; d < kDims; ++d) f[d] = sf[d * np + p0 + e];
            v = (unsigned long long)(unsigned)cell_of<kFineBits>(f, ext) << 32 | (unsigned)e;
        }
        key[e] = v;
    }
    __syncthreads();
    for (int size = 2; size <= kWindow; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const int a = 2 * tid - (tid & (stride - 1)), b = a + stride;
            const bool up = (a & size) == 0;
            const unsigned long long x = key[a], y = key[b];
            if ((x > y) == up) {
                key[a] = y;
                key[b] = x;
            }
            __syncthreads();
        }
    for (int d = 0; d <= kDims; ++d) {
        for (int e = tid; e < m; e += kWindow / 2)
            col[e] = d < kDims ? sf[d * np + p0 + e] : __int_as_float(sidx[p0 + e]);
        __syncthreads();
        for (int e = tid; e < m; e += kWindow / 2) {
            const float v = col[(unsigned)key[e]];
            if (d < kDims) sf[d * np + p0 + e] = v;
            else sidx[p0 + e] = __float_as_int(v);
        }
        __syncthreads();
    }
}

// Bounding box of every tile, a warp each: box[d * ntiles + t] = lo, then hi.
__global__ void k_tile_boxes(const float* __restrict__ sf, long long n, long long np, long long ntiles,
                             float* __restrict__ box) {
    const long long t = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    if (t >= ntiles) return;
    const int lane = threadIdx.x & 31;
    const long long p = min(t * kTile + lane, n - 1);
#pragma unroll
    for (int d = 0; d < kDims; ++d) {
        float lo = sf[d * np + p], hi = lo;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
            box[d * ntiles + t] = lo;
            box[(kDims + d) * ntiles + t] = hi;
        }
    }
}

// The search: a warp per tile of 32 queries, a lane per query. What bounds it
// is the distance evaluations of the tiles that are not skipped: about 18
// instructions per candidate for 32 queries. A candidate is first tested by a
// float32 sum of its squared differences, which is within 3e-7 of the float64
// distance; only those that pass (a margin of 2e-6 over the k-th distance) get
// the exact one and enter the lane's queue. Lists are unsorted in shared memory
// with their largest entry tracked; a replacement looks through the whole
// list, a chain of k shared-memory loads, so the lanes drain their queues
// together instead of one by one (1.6 ms a pass without the queues). Order of
// visits: the own tile and its neighbours on the curve, then
// tiles whose boxes overlap the queries', then the others, so that the k-th
// distances are tight by the time most boxes are looked at. 65536 points, k =
// 20 and 10: 7.8 ms a pass by tiles of 256 pixels in raster order, one query
// per thread with sorted lists in local memory; 0.9 ms here.
constexpr int kKnnWarps = 4;
constexpr float kMargin = 1.f - 2e-6f;
constexpr int kQueue = 8;            // a group of candidates adds at most kQueue / 2

__host__ __device__ constexpr size_t knn_warp_smem(int k) { return (size_t)(k + kQueue) * 32 * 12 + 32 * 32; }

__global__ void __launch_bounds__(kKnnWarps * 32) k_knn(const float* __restrict__ sf, const int* __restrict__ sidx,
                                                        const float* __restrict__ box, long long n, long long np,
                                                        long long ntiles, int k, int64_t* __restrict__ nbr) {
    extern __shared__ __align__(16) unsigned char knn_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long own = blockIdx.x * (long long)kKnnWarps + warp;
    if (own >= ntiles) return;
    // Candidates first (16-byte aligned), then the lists.
    float* cand = reinterpret_cast<float*>(knn_sm + warp * knn_warp_smem(k));
    double* D = reinterpret_cast<double*>(cand + 32 * 8) + lane;
    double* QD = D + k * 32;
    int* I = reinterpret_cast<int*>(QD - lane + kQueue * 32) + lane;
    int* QI = I + k * 32;
    const long long q = own * kTile + lane;
    const bool in = q < n;
    float qf[kDims], qlo[kDims], qhi[kDims];
    // A query with a feature that is not finite is infinitely far from every
    // point, so its list is the first k. Its lane goes along with a finite one
    // (a search of its own, which no tile can be left out of, kept the warp busy
    // with all of 65536 points for 14 ms a pass).
#pragma unroll
    for (int d = 0; d < kDims; ++d) qf[d] = sf[d * np + min(q, n - 1)];
    const unsigned finite = __ballot_sync(0xffffffffu, all_finite(qf));
    if (!finite) {
        if (in)
            for (int s = 0; s < k; ++s) nbr[(long long)sidx[q] * k + s] = s;
        return;
    }
    const long long with = min(finite >> lane & 1 ? q : own * kTile + __ffs(finite) - 1, n - 1);
#pragma unroll
    for (int d = 0; d < kDims; ++d) {
        qf[d] = sf[d * np + with];
        qlo[d] = box[d * ntiles + own];
        qhi[d] = box[(kDims + d) * ntiles + own];
    }
    int cnt = 0, maxpos = 0, maxI = 0;
    double maxD = 0.0;
    float thr = in ? __int_as_float(0x7f800000) : -1.f;     // bound of the k-th distance
    int qn = 0;
    auto drain = [&]() {
        for (int e = 0; __any_sync(0xffffffffu, e < qn); ++e) {
            if (e >= qn) continue;
            const double dist = QD[e * 32];
            const int ci = QI[e * 32];
            if (cnt < k) {
                D[cnt * 32] = dist;
                I[cnt * 32] = ci;
                if (cnt == 0 || dist > maxD || (dist == maxD && ci > maxI)) {
                    maxD = dist;
                    maxI = ci;
                    maxpos = cnt;
                }
                ++cnt;
            } else if (dist < maxD || (dist == maxD && ci < maxI)) {
                D[maxpos * 32] = dist;
                I[maxpos * 32] = ci;
                maxD = D[0];
                maxpos = 0;
                bool tie = false;
#pragma unroll 4
                for (int s = 1; s < k; ++s) {
                    const double v = D[s * 32];
                    tie = v > maxD ? false : (tie || v == maxD);
                    if (v > maxD) {
                        maxD = v;
                        maxpos = s;
                    }
                }
                maxI = I[maxpos * 32];
                if (tie)                                  // the largest index among the largest
                    for (int s = 0; s < k; ++s)
                        if (D[s * 32] == maxD && I[s * 32] > maxI) {
                            maxI = I[s * 32];
                            maxpos = s;
                        }
            }
        }
        qn = 0;
        if (cnt == k && in) thr = __double2float_ru(maxD);
    };
    auto visit = [&](long long t) {
        __syncwarp();
        const long long c0 = t * kTile;
        const int m = (int)min((long long)kTile, n - c0);
        if (lane < m) {
            const long long c = c0 + lane;
            *reinterpret_cast<float4*>(cand + lane * 8) = make_float4(sf[c], sf[np + c], sf[2 * np + c], sf[3 * np + c]);
            cand[lane * 8 + 4] = sf[4 * np + c];
            reinterpret_cast<int*>(cand)[lane * 8 + 5] = sidx[c];
        }
        __syncwarp();
        for (int cg = 0; cg < m; cg += kQueue / 2) {
#pragma unroll
            for (int u = 0; u < kQueue / 2; ++u) {
                const int c = cg + u;
                const float4 a = *reinterpret_cast<const float4*>(cand + c * 8);
                const float2 e = *reinterpret_cast<const float2*>(cand + c * 8 + 4);
                const float d0 = __fsub_rn(qf[0], a.x), d1 = __fsub_rn(qf[1], a.y), d2 = __fsub_rn(qf[2], a.z);
                const float d3 = __fsub_rn(qf[3], a.w), d4 = __fsub_rn(qf[4], e.x);
                const float p0 = __fmul_rn(d0, d0), p1 = __fmul_rn(d1, d1), p2 = __fmul_rn(d2, d2);
                const float p3 = __fmul_rn(d3, d3), p4 = __fmul_rn(d4, d4);
                if (c >= m || (p0 + p1 + p2 + p3 + p4) * kMargin > thr) continue;
                double dist = (double)p0;
                dist = __dadd_rn(dist, (double)p1);
                dist = __dadd_rn(dist, (double)p2);
                dist = __dadd_rn(dist, (double)p3);
                dist = __dadd_rn(dist, (double)p4);
                // The lists' order has no place for NaN: as infinite, it leaves
                // finite queries' lists alone.
                QD[qn * 32] = dist == dist ? dist : __longlong_as_double(0x7ff0000000000000ll);
                QI[qn * 32] = __float_as_int(e.y);
                ++qn;
            }
            if (__any_sync(0xffffffffu, qn >= kQueue / 2)) drain();
        }
        if (__any_sync(0xffffffffu, cnt < k && in)) drain();
    };
    // Whether any query of the warp may find a neighbour in tile t.
    auto wanted = [&](long long t) {
        float lb = 0.f;
#pragma unroll
        for (int d = 0; d < kDims; ++d) {
            const float e = fmaxf(fmaxf(box[d * ntiles + t] - qf[d], qf[d] - box[(kDims + d) * ntiles + t]), 0.f);
            lb += e * e;
        }
        return __any_sync(0xffffffffu, in && !(lb * kMargin > thr));
    };
    constexpr int kNear = 2;
    visit(own);
    for (int d = 1; d <= kNear; ++d) {
        if (own - d >= 0 && wanted(own - d)) visit(own - d);
        if (own + d < ntiles && wanted(own + d)) visit(own + d);
    }
    for (int sweep = 0; sweep < 2; ++sweep) {
        for (long long t0 = 0; t0 < ntiles; t0 += 32) {
            float T = thr;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) T = fmaxf(T, __shfl_xor_sync(0xffffffffu, T, o));
            const long long t = t0 + lane;
            bool take = false;
            if (t < ntiles && (t < own - kNear || t > own + kNear)) {
                float gap = 0.f;
#pragma unroll
                for (int d = 0; d < kDims; ++d) {
                    const float e = fmaxf(fmaxf(box[d * ntiles + t] - qhi[d], qlo[d] - box[(kDims + d) * ntiles + t]), 0.f);
                    gap += e * e;
                }
                take = sweep == 0 ? gap == 0.f : gap != 0.f && !(gap * kMargin > T);
            }
            unsigned bits = __ballot_sync(0xffffffffu, take);
            while (bits) {
                const int b = __ffs(bits) - 1;
                bits &= bits - 1;
                if (wanted(t0 + b)) visit(t0 + b);
            }
        }
    }
    drain();
    if (in) {
        const long long i = sidx[q];
#pragma unroll
        for (int d = 0; d < kDims; ++d) qf[d] = sf[d * np + q];
        const bool found = all_finite(qf);
        for (int s = 0; s < k; ++s) nbr[i * k + s] = !found ? s : s < cnt ? I[s * 32] : i;
    }
}

struct Pass {
    const int64_t* nbr;  // (n, k)
    const float* f;      // (n, 5)
    int k;
};
struct Passes {
    Pass p[4];
    int np;
    int soft;
};

__device__ __forceinline__ double edge_value(const Passes& P, int pi, long long i, long long j) {
    if (!P.soft) return 1.0;
    const float* a = P.p[pi].f + i * kDims;
    const float* b = P.p[pi].f + j * kDims;
    float s = 0.f;
    for (int d = 0; d < kDims; ++d) s = __fadd_rn(s, fabsf(__fsub_rn(a[d], b[d])));
    return __dsub_rn(1.0, (double)__fdiv_rn(s, (float)kDims));
}

// Whether pixel q is in one of its own lists. It is not where more than k
// pixels are equal to it and have smaller indices; its row then gets an entry
// (q, q) of weight zero, which L = I - D^-1 W needs for its diagonal.
__device__ __forceinline__ bool lists_itself(const Passes& P, long long q) {
    for (int pi = 0; pi < P.np; ++pi)
        for (int e = 0; e < P.p[pi].k; ++e)
            if (P.p[pi].nbr[q * P.p[pi].k + e] == q) return true;
    return false;
}

// Entries of every row: its own, and one for each edge q -> j that gives row
// j one.
__global__ void k_degree(Passes P, long long n, int kt, int64_t* cap) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= n) return;
    for (int pi = 0; pi < P.np; ++pi)
        for (int e = 0; e < P.p[pi].k; ++e)
            atomicAdd((unsigned long long*)(cap + P.p[pi].nbr[q * P.p[pi].k + e]), 1ull);
    atomicAdd((unsigned long long*)(cap + q), (unsigned long long)(kt + !lists_itself(P, q)));
}

// Scatter: own neighbours at the start of the row's slots, the others (reverse
// edges, the zero on the diagonal) after them (slot claimed with an atomic
// counter).
__global__ void k_scatter(Passes P, long long n, int kt, const int64_t* off, int64_t* fillc,
                          int64_t* cols, double* vals) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q >= n) return;
    long long o = off[q];
    auto put = [&](long long row, long long col, double v) {
        const long long slot = off[row] + kt + (long long)atomicAdd((unsigned long long*)(fillc + row), 1ull);
        cols[slot] = col;
        vals[slot] = v;
    };
    for (int pi = 0; pi < P.np; ++pi)
        for (int e = 0; e < P.p[pi].k; ++e) {
            const long long j = P.p[pi].nbr[q * P.p[pi].k + e];
            const double v = edge_value(P, pi, q, j);
            cols[o] = j;
            vals[o] = v;
            ++o;
            put(j, q, v);
        }
    if (!lists_itself(P, q)) put(q, q, 0.0);
}

// Order-preserving map of doubles to unsigned. A total order: NaN, which the
// soft kernel gives where a feature is not finite, has its place in it too.
__device__ __forceinline__ unsigned long long ordered64(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return u >> 63 ? ~u : u | 1ull << 63;
}
__device__ __forceinline__ double unordered64(unsigned long long u) {
    return __longlong_as_double((long long)(u >> 63 ? u & ~(1ull << 63) : ~u));
}

// Sort each row by (column, value), merge duplicates (sum in that order),
// count the unique columns. A warp per row: entries find their ranks by
// counting the smaller ones in shared memory (rows hold about 2 kt entries;
// one thread per row shifting entries in global memory took 1.6 ms for 65536
// rows); the ranks are a permutation because (column, ordered64, position) is
// a total order. A row of more than kSortMax entries, one that many others
// list, takes its whole CTA, of more than kSortWarps times that one thread.
constexpr int kSortMax = 256, kSortWarps = 4;
__host__ __device__ constexpr size_t sort_warp_smem() { return (size_t)kSortMax * 24; }

__device__ void sort_merge_one(long long a, long long m, int64_t* cols, double* vals, int64_t* ucount) {
    for (long long s = 1; s < m; ++s) {
        const int64_t c = cols[a + s];
        const double v = vals[a + s];
        long long t = s - 1;
        while (t >= 0 && (cols[a + t] > c || (cols[a + t] == c && vals[a + t] > v))) {
            cols[a + t + 1] = cols[a + t];
            vals[a + t + 1] = vals[a + t];
            --t;
        }
        cols[a + t + 1] = c;
        vals[a + t + 1] = v;
    }
    long long u = 0;
    for (long long s = 0; s < m; ++s) {
        if (s > 0 && cols[a + s] == cols[a + u - 1]) {
            vals[a + u - 1] = __dadd_rn(vals[a + u - 1], vals[a + s]);
        } else {
            cols[a + u] = cols[a + s];
            vals[a + u] = vals[a + s];
            ++u;
        }
    }
    *ucount = u;
}

// m entries at a by `nthr` threads (tid among them), with shared memory for
// `room` entries and a barrier for those threads.
template <typename Sync>
__device__ __forceinline__ void sort_merge_row(long long a, int m, int tid, int nthr, unsigned char* sm, int room,
                                               int64_t* cols, double* vals, int64_t* ucount, Sync sync) {
    unsigned long long* v0 = reinterpret_cast<unsigned long long*>(sm);   // ordered64
    double* v1 = reinterpret_cast<double*>(v0 + room);
    int* c0 = reinterpret_cast<int*>(v1 + room);
    int* c1 = c0 + room;
    const int m4 = (m + 3) & ~3;                       // <= room
    for (int e = tid; e < m4; e += nthr) {
        c0[e] = e < m ? (int)cols[a + e] : 0x7fffffff;
        if (e < m) v0[e] = ordered64(vals[a + e]);
    }
    sync();
    for (int e = tid; e < m; e += nthr) {
        const int c = c0[e];
        const unsigned long long v = v0[e];
        int rank = 0;
        for (int t = 0; t < m4; t += 4) {
            const int4 k = *reinterpret_cast<const int4*>(c0 + t);
            rank += (k.x < c) + (k.y < c) + (k.z < c) + (k.w < c);
            if (k.x == c || k.y == c || k.z == c || k.w == c)
                for (int q = t; q < t + 4; ++q)
                    rank += c0[q] == c && (v0[q] < v || (v0[q] == v && q < e));
        }
        c1[rank] = c;
        v1[rank] = unordered64(v);
    }
    sync();
    // The first warp merges.
    if (tid >= 32) return;
    int u = 0;
    for (int e0 = 0; e0 < m; e0 += 32) {
        const int e = e0 + tid;
        const bool head = e < m && (e == 0 || c1[e] != c1[e - 1]);
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        if (head) {
            double s = v1[e];
            for (int t = e + 1; t < m && c1[t] == c1[e]; ++t) s = __dadd_rn(s, v1[t]);
            const int at = u + __popc(heads & ((1u << tid) - 1u));
            cols[a + at] = c1[e];
            vals[a + at] = s;
        }
        u += __popc(heads);
    }
    if (tid == 0) *ucount = u;
}

__global__ void __launch_bounds__(kSortWarps * 32) k_sort_merge(long long n, const int64_t* off, const int64_t* cap,
                                                                int64_t* cols, double* vals, int64_t* ucount) {
    extern __shared__ __align__(16) unsigned char sort_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long i0 = blockIdx.x * (long long)kSortWarps;
    if (i0 + warp < n && cap[i0 + warp] <= kSortMax)
        sort_merge_row(off[i0 + warp], (int)cap[i0 + warp], lane, 32, sort_sm + warp * sort_warp_smem(), kSortMax,
                       cols, vals, ucount + i0 + warp, [] { __syncwarp(); });
    for (int r = 0; r < kSortWarps; ++r) {
        if (i0 + r >= n || cap[i0 + r] <= kSortMax) continue;
        __syncthreads();
        if (cap[i0 + r] <= kSortMax * kSortWarps)
            sort_merge_row(off[i0 + r], (int)cap[i0 + r], threadIdx.x, kSortWarps * 32, sort_sm,
                           kSortMax * kSortWarps, cols, vals, ucount + i0 + r, [] { __syncthreads(); });
        else if (threadIdx.x == 0)
            sort_merge_one(off[i0 + r], cap[i0 + r], cols, vals, ucount + i0 + r);
    }
}

// L = I - diag(1 / rowsum(W)) W into the final CSR, a warp per row; the row
// sum in order (every lane adds the entries it is handed).
__global__ void __launch_bounds__(256) k_normalize(long long n, const int64_t* off, const int64_t* rowptr,
                                                   const int64_t* wcols, const double* wvals, int64_t* cols,
                                                   double* vals) {
    const long long i = blockIdx.x * 8ll + (threadIdx.x >> 5);
    if (i >= n) return;
    const int lane = threadIdx.x & 31;
    const long long a = off[i], b = rowptr[i], u = rowptr[i + 1] - b;
    double s = 0.0;
    for (long long t0 = 0; t0 < u; t0 += 32) {
        const double v = t0 + lane < u ? wvals[a + t0 + lane] : 0.0;
        const int m = (int)min(32ll, u - t0);
        for (int t = 0; t < m; ++t) s = __dadd_rn(s, __shfl_sync(0xffffffffu, v, t));
    }
    const double fct = __ddiv_rn(1.0, s);
    for (long long t = lane; t < u; t += 32) {
        const long long j = wcols[a + t];
        const double wp = __dmul_rn(fct, wvals[a + t]);
        cols[b + t] = j;
        vals[b + t] = (j == i) ? __dsub_rn(1.0, wp) : -wp;
    }
}

}  // namespace knn
}  // namespace pmb

using namespace pmb::knn;

static long long padded(long long n) { return (n + 31) / 32 * 32; }
// int64 elements of the search: extent, cell of every point, ordered points
// and their indices, boxes, buckets and the scan's chunk sums.
static long long search_elems(long long n) {
    const long long np = padded(n), ntiles = np / kTile;
    return 8 + np / 2 + kDims * np / 2 + np / 2 + kDims * ntiles + kCells + 1 + kCells / 1024 + 4;
}

// Scratch elements (int64) for pmb_launch_knn with n pixels, total
// neighbours per pixel kt and passes np: features, neighbour lists, row
// capacities / offsets / fill counters / unique counts, and the unmerged
// W (2 n kt entries and at most n zeros on the diagonal, columns + values).
// The search's ordered points, boxes and buckets share the space of W, which is
// filled after it.
int64_t pmb_launch_knn_scratch(long long n, int kt, int np) {
    if (n <= 0 || kt <= 0 || np <= 0 || np > 4) return -1;
    const long long feat = (n * kDims * np * 4 + 7) / 8;  // floats -> int64 slots
    return feat + n * kt + 4 * (n + 1) + ((n + 1) + 1023) / 1024 + 2 +
           std::max(2 * (2 * n * kt + n), search_elems(n));
}

// Two calls on the same scratch and rowptr. First (cols / vals null): the
// neighbour search and the merged rows of W; writes rowptr and the number of
// stored entries of L to *nnz_out (synchronises the stream once). Second
// (cols / vals of *nnz_out entries): L from the state the first call left.
int pmb_launch_knn(const double* image, int h, int w, const int* ks, const double* dws, int np,
                   int soft, int64_t* scratch, int64_t* rowptr, int64_t* cols, double* vals,
                   int64_t* nnz_out, cudaStream_t st) {
    const long long n = (long long)h * w;
    if (!image || !ks || !dws || np <= 0 || np > 4 || !scratch || !rowptr || n <= 0) return -2;
    int kt = 0;
    for (int p = 0; p < np; ++p) {
        if (ks[p] <= 0 || ks[p] > kMaxK || ks[p] > n) return -2;
        kt += ks[p];
    }
    float* feat = (float*)scratch;
    int64_t* s = scratch + (n * kDims * np * 4 + 7) / 8;
    int64_t* nbr = s;
    s += n * kt;
    int64_t* cap = s;
    s += n + 1;
    int64_t* off = s;
    s += n + 1;
    int64_t* fillc = s;
    s += n + 1;
    int64_t* ucount = s;
    s += n + 1;
    int64_t* chunk = s;
    s += ((n + 1) + 1023) / 1024 + 2;
    int64_t* wcols = s;
    s += 2 * n * kt + n;
    double* wvals = (double*)s;
    const int blocks = (int)((n + 255) / 256);
    if (cols && vals) {
        k_normalize<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(n, off, rowptr, wcols, wvals, cols, vals);
        return pmb::launch_status() ? 1 : 0;
    }
    Passes P{};
    P.np = np;
    P.soft = soft;
    int64_t* nb = nbr;
    const long long npad = padded(n), ntiles = npad / kTile;
    unsigned* ext = (unsigned*)wcols;
    int* cell = (int*)(wcols + 8);
    float* sf = (float*)(cell + npad);
    int* sidx = (int*)(sf + kDims * npad);
    float* boxes = (float*)(sidx + npad);
    int64_t* buckets = (int64_t*)(boxes + 2 * kDims * ntiles);
    int64_t* bchunk = buckets + kCells + 1;
    int kmax = 0;
    for (int p = 0; p < np; ++p) kmax = std::max(kmax, ks[p]);
    if (kKnnWarps * knn_warp_smem(kmax) > 48 * 1024 &&
        cudaFuncSetAttribute(k_knn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(kKnnWarps * knn_warp_smem(kmax))) != cudaSuccess)
        return 1;
    for (int p = 0; p < np; ++p) {
        float* fp = feat + (long long)p * n * kDims;
        if (cudaMemsetAsync(ext, 0, 64, st) != cudaSuccess ||
            cudaMemsetAsync(buckets, 0, (kCells + 1) * sizeof(int64_t), st) != cudaSuccess)
            return 1;
        k_features<<<blocks, 256, 0, st>>>(image, h, w, dws[p], fp, ext);
        k_cell_count<<<blocks, 256, 0, st>>>(fp, n, ext, cell, buckets);
        if (pmb_scan_exclusive(buckets, kCells, bchunk, buckets + kCells, st)) return 1;
        k_reorder<<<blocks, 256, 0, st>>>(fp, n, npad, cell, buckets, sf, sidx);
        k_refine<<<(unsigned)((n + kWindow - 1) / kWindow), kWindow / 2, 0, st>>>(n, npad, ext, sf, sidx);
        k_tile_boxes<<<(unsigned)((ntiles + 7) / 8), 256, 0, st>>>(sf, n, npad, ntiles, boxes);
        k_knn<<<(unsigned)((ntiles + kKnnWarps - 1) / kKnnWarps), kKnnWarps * 32,
                kKnnWarps * knn_warp_smem(ks[p]), st>>>(sf, sidx, boxes, n, npad, ntiles, ks[p], nb);
        P.p[p] = Pass{nb, fp, ks[p]};
        nb += n * ks[p];
    }
    if (cudaMemsetAsync(cap, 0, 3 * (n + 1) * sizeof(int64_t), st) != cudaSuccess) return 1;
    k_degree<<<blocks, 256, 0, st>>>(P, n, kt, cap);
    cudaMemcpyAsync(off, cap, n * sizeof(int64_t), cudaMemcpyDeviceToDevice, st);
    if (pmb_scan_exclusive(off, n, chunk, off + n, st)) return 1;
    cudaMemsetAsync(fillc, 0, (n + 1) * sizeof(int64_t), st);
    k_scatter<<<blocks, 256, 0, st>>>(P, n, kt, off, fillc, wcols, wvals);
    k_sort_merge<<<(unsigned)((n + kSortWarps - 1) / kSortWarps), kSortWarps * 32, kSortWarps * sort_warp_smem(), st>>>(
        n, off, cap, wcols, wvals, ucount);
    cudaMemcpyAsync(rowptr, ucount, n * sizeof(int64_t), cudaMemcpyDeviceToDevice, st);
    if (pmb_scan_exclusive(rowptr, n, chunk, rowptr + n, st)) return 1;
    int64_t nnz = 0;
    cudaMemcpyAsync(&nnz, rowptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return 1;
    if (nnz_out) *nnz_out = nnz;
    return pmb::launch_status() ? 1 : 0;
}
