// Thresholded incomplete Cholesky factorisation and its triangular solves.
//
// Restates pymatting/preconditioner/ichol.py:
//   _ichol :6-113           column-by-column factorisation with absolute and
//                           relative discard thresholds, diagonal compensation
//                           of discarded entries, failure codes -1 (not
//                           positive definite) / -2 (more than max_nnz);
//   _backsub_L_csc_inplace  :116-129  and  _backsub_LT_csc_inplace :132-145.
//
// The factorisation is inherently sequential over columns (column j needs
// every column k < j that has a kept entry in row j). Three kernels make it,
// with the reference's keep and discard rules, every update of an entry in
// ascending k and one rounding each for product and difference, so their
// factors are identical:
//   k_ichol_factor_pipe     left-looking, a pipeline of the warps of one CTA:
//                           bandwidths up to 1024 (below);
//   k_ichol_factor_cluster  right-looking, the band front in a cluster's shared
//                           memory: wide bands with long columns
//                           (ichol_cluster.cu);
//   k_ichol_factor          right-looking, the front in global memory, one CTA:
//                           the widest bands. When column k is final, its kept
//                           entries update the pending columns k+1 .. k+B
//                           directly (B = bandwidth of A; fill never leaves
//                           the envelope). Per column, warp 0 does the serial
//                           part with warp ballots (candidate rows, pivot,
//                           thresholding, compaction), then the whole CTA does
//                           the pair updates while the last warp recycles the
//                           column's front slot: two block barriers a column.
//
// The factor's dependency levels (level[i] = 1 + max level of the columns
// that update row i) fall out of the factorisation for free and drive the
// level-scheduled triangular solves: one thread per row inside a level,
// rows subtract their terms in the reference's order, levels separated by
// block barriers (single CTA: the systems this preconditioner is used on
// are the compressed unknown regions, tens of thousands of rows).
#include "pm_common.cuh"
#include "ichol.cuh"
#include "tma.cuh"

namespace pmb {

constexpr int kIcholThreads = 1024;
constexpr int kIcholChunks = 8;      // front columns of up to 256 rows load in one burst
constexpr size_t kFactorSmem = 227 * 1024 - 256;
constexpr int64_t kIcholSmemRows = 27 * 1024;   // x of the shared-memory solve: 216 KB

// Per-column statistics of A (lower part, CSC): diagonal (+ shift), sum of
// |A[j:, j]| for the relative threshold, and the largest i - j.
__global__ void k_ichol_init(int64_t n, const int64_t* __restrict__ Ap,
                             const int64_t* __restrict__ Ar, const double* __restrict__ Av,
                             double shift, double* d, double* rsum, int* level,
                             unsigned long long* band) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    double dj = shift, rj = 0.0;
    int64_t bmax = 0;
    for (int64_t k = Ap[j]; k < Ap[j + 1]; ++k) {
        const int64_t i = Ar[k];
        if (i == j) dj += Av[k];
        if (i >= j) rj += fabs(Av[k]);
        if (i > j && Av[k] != 0.0 && i - j > bmax) bmax = i - j;
    }
    d[j] = dj;
    rsum[j] = rj;
    level[j] = 0;
    if (bmax > 0) atomicMax(band, (unsigned long long)bmax);
}

// Load column j of A (entries below the diagonal with non-zero value) into
// its front slot. The slot was cleared beforehand.
__device__ __forceinline__ void load_column(int64_t j, int64_t W, const int64_t* __restrict__ Ap,
                                            const int64_t* __restrict__ Ar,
                                            const double* __restrict__ Av, double* F,
                                            uint8_t* pat) {
    const int64_t slot = (j % W) * W;
    for (int64_t k = Ap[j] + threadIdx.x; k < Ap[j + 1]; k += blockDim.x) {
        const int64_t i = Ar[k];
        const double v = Av[k];
        if (i > j && v != 0.0) {
            // Canonical input has one entry per (i, j): no two threads
            // write the same offset.
            F[slot + (i - j)] += v;
            pat[slot + (i - j)] = 1;
        }
    }
}

// The front in global memory. One CTA. Front F / pat: W x W (W = B + 1), slot of
// column j = j % W, entry (i, j) at offset i - j. cand / kept: scratch of
// at least W entries each.
__global__ void __launch_bounds__(kIcholThreads)
k_ichol_factor(int64_t n, int64_t W, const int64_t* __restrict__ Ap,
               const int64_t* __restrict__ Ar, const double* __restrict__ Av, double* d,
               const double* __restrict__ rsum, int* level, double* F, uint8_t* pat, int* cand,
               double* keptv, int64_t* kepti, int64_t* Lp, int64_t* Lr, double* Lv,
               int64_t cap, double discard, int64_t max_nnz, double rel_discard, int diag_keep,
               int64_t* result) {
    __shared__ int64_t s_nnz;
    __shared__ int s_m, s_fail;
    __shared__ double s_keptv[kIcholChunks * 32];     // kept entries of the column
    __shared__ int64_t s_kepti[kIcholChunks * 32];

    // Initial front: columns 0 .. W-1.
    for (int64_t j = 0; j < W && j < n; ++j) load_column(j, W, Ap, Ar, Av, F, pat);
    if (threadIdx.x == 0) {
        s_nnz = 0;
        s_fail = 0;
        Lp[0] = 0;
    }
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t j = 0; j < n; ++j) {
        const int64_t slot = (j % W) * W;
        // Warp 0: the serial part of column j, warp-synchronous. Offsets
        // o = 1 + lane + 32 k: chunk k, lane order = ascending rows, the
        // order in which the reference sorts its candidates (ichol.py:87-89).
        // The pattern flags and front values of the first kIcholChunks
        // chunks, the pivot and the threshold are loaded in one burst.
        if (warp == 0) {
            bool flag[kIcholChunks];
            double aval[kIcholChunks];
#pragma unroll
            for (int k = 0; k < kIcholChunks; ++k) {
                const int64_t o = 1 + lane + 32 * k;
                flag[k] = o < W && j + o < n && pat[slot + o];
                aval[k] = flag[k] ? F[slot + o] : 0.0;
            }
            const double dj = d[j];
            const double rel = rel_discard * rsum[j];
            int cn = 0;
#pragma unroll
            for (int k = 0; k < kIcholChunks; ++k) cn += __popc(__ballot_sync(0xffffffffu, flag[k]));
            for (int64_t base = 1 + 32 * kIcholChunks; base < W; base += 32) {   // wide bands
                const int64_t o = base + lane;
                cn += __popc(__ballot_sync(0xffffffffu, o < W && j + o < n && pat[slot + o]));
            }
            int fail = 0;
            const int64_t nnz = s_nnz;
            if (!(dj > 0.0)) fail = -1;                                   // ichol.py:80-81
            else if (nnz + 1 + cn > max_nnz || nnz + 1 + cn > cap) fail = -2;   // ichol.py:82-83
            int kept = 0;
            int64_t nnz0 = nnz + 1;
            if (!fail) {
                const double sj = sqrt(dj);
                if (lane == 0) {
                    d[j] = sj;
                    Lv[nnz] = sj;
                    Lr[nnz] = j;
                }
                auto take = [&](bool fl, double a, int64_t o) {
                    bool keep = false;
                    double L = 0.0;
                    const int64_t i = j + o;
                    if (fl) {
                        L = a / sj;
                        if (diag_keep) d[i] -= L * L;
                        keep = fabs(L) > discard && fabs(a) > rel;
                        if (keep && !diag_keep) d[i] -= L * L;
                    }
                    const unsigned mask = __ballot_sync(0xffffffffu, keep);
                    if (keep) {
                        const int pos = kept + __popc(mask & ((1u << lane) - 1u));
                        Lv[nnz0 + pos] = L;
                        Lr[nnz0 + pos] = i;
                        keptv[pos] = L;
                        kepti[pos] = i;
                        if (pos < kIcholChunks * 32) {
                            s_keptv[pos] = L;
                            s_kepti[pos] = i;
                        }
                    }
                    kept += __popc(mask);
                };
#pragma unroll
                for (int k = 0; k < kIcholChunks; ++k) take(flag[k], aval[k], 1 + lane + 32 * k);
                for (int64_t base = 1 + 32 * kIcholChunks; base < W; base += 32) {
                    const int64_t o = base + lane;
                    const bool fl = o < W && j + o < n && pat[slot + o];
                    take(fl, fl ? F[slot + o] : 0.0, o);
                }
            }
            if (lane == 0) {
                s_fail = fail;
                if (!fail) {
                    s_m = kept;
                    s_nnz = nnz0 + kept;
                    Lp[j + 1] = nnz0 + kept;
                }
            }
        }
        __syncthreads();
        if (s_fail) break;
        const int m = s_m;
        // Levels of the rows this column feeds.
        const int lj = level[j] + 1;
        for (int q = threadIdx.x; q < m; q += blockDim.x) {
            const int64_t i = m <= kIcholChunks * 32 ? s_kepti[q] : kepti[q];
            if (level[i] < lj) level[i] = lj;
        }
        // Right-looking update of the pending columns: for kept rows
        // ia > ib, F[ib][ia - ib] -= L_ia L_ib, one pair per thread. Rows ib
        // lie in (j, j + W), so no update touches slot j.
        const bool shared_list = m <= kIcholChunks * 32;
        const double* kv = shared_list ? s_keptv : keptv;
        const int64_t* ki = shared_list ? s_kepti : kepti;
        const int64_t pairs = (int64_t)m * (m - 1) / 2;
        for (int64_t p = threadIdx.x; p < pairs; p += blockDim.x) {
            // Invert p = a (a - 1) / 2 + b with 0 <= b < a.
            int64_t a = (int64_t)((1.0 + sqrt(1.0 + 8.0 * (double)p)) * 0.5);
            while (a * (a - 1) / 2 > p) --a;
            while ((a + 1) * a / 2 <= p) ++a;
            const int64_t b = p - a * (a - 1) / 2;
            const int64_t ia = ki[a], ib = ki[b];
            const int64_t off = ((ib % W) * W) + (ia - ib);
            F[off] -= kv[a] * kv[b];
            pat[off] = 1;
        }
        // Meanwhile the last warp recycles slot j for column j + W (clear,
        // then load; ordered within the warp).
        if (warp == (int)(blockDim.x >> 5) - 1) {
            for (int64_t o = lane; o < W; o += 32) {
                F[slot + o] = 0.0;
                pat[slot + o] = 0;
            }
            __syncwarp();
            if (j + W < n) {
                const int64_t jn = j + W;
                for (int64_t k = Ap[jn] + lane; k < Ap[jn + 1]; k += 32) {
                    const int64_t i = Ar[k];
                    const double v = Av[k];
                    if (i > jn && v != 0.0) {
                        F[slot + (i - jn)] += v;
                        pat[slot + (i - jn)] = 1;
                    }
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *result = s_fail ? (int64_t)s_fail : s_nnz;
}

// ---------------------------------------------------------------------------
// The same factorisation, left-looking, as a pipeline of the warps of one CTA.
//
//   walkers   the other warps, column j on walker j mod their number: A's entries
//             of column j into an accumulator of W values in shared memory,
//             then minus L_jk L_ik for every column k < j - kLag with a kept
//             entry in row j, in ascending k, as those columns are done.
//   finishers kFin warps, every column in turn, one offset below the pivot per
//             lane (and chunk): the last kLag columns' terms from dense copies
//             in shared memory, one quotient, thresholds, diagonal update.
//   pivot     one warp: the next pivot's root and its reciprocal, and the wait
//             for the walker of the column after that.
//   publishers kFin warps: the entries' places in L and in their rows' lists.
//
// What stays on the chain from one column to the next is the quotient, the
// root and two barriers of the finishers, the publishers and the pivot warp;
// about 1,700 cycles, where the front spread over a cluster's shared memory
// (every CTA reading, dividing and compacting the pivot column, then a cluster
// barrier) took 4,300. 11,407 columns (W = 232), 45 entries kept in each: 25.9
// -> 10.2 ms; without publishers of their own (the finishers writing L) 10.9.
// The walkers' reads of L bound it now: with 11 of them 13.9 ms, 15: 12.1.
//
// L itself, in global memory, is what the walkers read (one CTA: its columns
// come from L1 or L2), so nothing limits the number of entries. Row i's list,
// in ascending columns, has the place in L of each kept entry of row i, how
// many entries of its column follow, and its offset; entries nearer than
// kLag to the diagonal are not listed. Every subtraction of an entry runs in
// ascending k with one rounding for the product and one for the difference, as
// in the kernels above: the factors are identical.
//
// An accumulator or a dense copy that holds -0.0 has no entry (an entry is
// never -0.0: A's are non-zero and every update ends with + 0.0).
// ---------------------------------------------------------------------------

// Warps for `fin` finishers: as many publishers, the pivot, and walkers.
__host__ __device__ constexpr int pipe_warps(int fin) { return fin <= 6 ? 28 : 32; }
__host__ __device__ constexpr int pipe_walkers(int fin) { return pipe_warps(fin) - 1 - 2 * fin; }
constexpr int kLag = 4;
constexpr int kDense = 8;             // dense columns kept (a power of two above kLag)
constexpr int kPipeMaxChunks = 32;    // 32-offset chunks of a column: W <= 1025
constexpr int kBatch = 2;             // nodes whose entries a walker has in flight
constexpr int kPipeStop = 0x7fffffff;
constexpr int64_t kPipeMax = (int64_t)1 << 30;

struct PipeLayout {
    int Wp;
    size_t o_dense, o_d, o_lev, o_pos, o_cnt, bytes;
};

__host__ __device__ inline PipeLayout pipe_layout(int64_t W, int walkers) {
    PipeLayout L;
    L.Wp = (int)((W + kLag + 7) & ~(int64_t)7);
    size_t o = (size_t)walkers * L.Wp * 8;
    L.o_dense = o; o += (size_t)kDense * L.Wp * 8;
    L.o_d = o;     o += (size_t)L.Wp * 8;
    L.o_lev = o;   o += (size_t)L.Wp * 4;
    L.o_pos = o;   o += (size_t)L.Wp * 4;
    L.o_cnt = o;   o += (size_t)L.Wp * 4;
    L.bytes = (o + 15) & ~(size_t)15;
    return L;
}

__device__ __forceinline__ void st_release(int* p, int v) {
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}

template <int FIN>
__device__ __forceinline__ void pipe_barrier(int id) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(32 * (2 * FIN + 1)) : "memory");
}

// Exponents for which a quotient by `pipe_quotient` cannot leave the normal
// range, nor its remainders.
__device__ __forceinline__ bool mid_range(double x) {
    const int e = (__double2hiint(x) >> 20) & 0x7ff;
    return e > 523 && e < 1523;
}

// Roots whose reciprocal `y` in the pivot warp serves `pipe_quotient`.
__device__ __forceinline__ bool root_range(double s) {
    return mid_range(s) && (__double2hiint(s) & 0xfffff) != 0xfffff;
}

// a / b, correctly rounded, from y within (1/2 + 2^-48) ulp of 1 / b: a y is
// within two ulp, one correction by its remainder makes it faithful and a
// second one, whose remainder is exact, the rounded quotient (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990). With the significand of b at beta 2^53, beta < 1, the corrected value
// is within 2^-54 beta (1 + 2^-47) ulp of a / b before its rounding, and a / b
// is at least 2^-54 / beta ulp from a midpoint of two doubles; the range of b
// leaves out the beta next to 1. For a zero or in the range above.
__device__ __forceinline__ double pipe_quotient(double a, double b, double y) {
    double q = a * y;
    q = __fma_rn(__fma_rn(-q, b, a), y, q);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

__device__ __forceinline__ bool has_entry(double a) {
    return __double_as_longlong(a) != (long long)0x8000000000000000ull;
}

// list: W x W nodes, row i's at slot i mod W; a node is the entry's place in
// L and (entries of its column after it) << 16 | offset.
template <int kFin, int M>
__global__ void __launch_bounds__(32 * pipe_warps(kFin), 1)
k_ichol_factor_pipe(int n, int W, const int64_t* __restrict__ Ap, const int64_t* __restrict__ Ar,
                    const double* __restrict__ Av, const double* __restrict__ d0,
                    const double* __restrict__ rsum, int* level, int64_t* Lp, int64_t* Lr, double* Lv,
                    int2* list, uint16_t* offs, int64_t cap, double discard, int64_t max_nnz, double rel_discard,
                    int diag_keep, int64_t* result, uint32_t limit, int look_cols, int look_end, int64_t dense_nnz) {
    extern __shared__ __align__(16) unsigned char pipe_smem[];
    constexpr int kWalkers = pipe_walkers(kFin);
    __shared__ __align__(16) int s_count[2][kFin * M];  // candidates << 16 | kept, per chunk
    __shared__ double s_dj, s_sj, s_y;
    __shared__ int s_ready[kWalkers];          // column whose accumulator is ready
    __shared__ int s_done, s_stop;
    __shared__ int64_t s_result;
    const PipeLayout Ly = pipe_layout(W, kWalkers);
    const int Wp = Ly.Wp;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned all = 0xffffffffu, lt = (1u << lane) - 1u;
    double* accs = reinterpret_cast<double*>(pipe_smem);
    double* dense = reinterpret_cast<double*>(pipe_smem + Ly.o_dense);
    double* dl = reinterpret_cast<double*>(pipe_smem + Ly.o_d);
    int* lev = reinterpret_cast<int*>(pipe_smem + Ly.o_lev);
    int* rowpos = reinterpret_cast<int*>(pipe_smem + Ly.o_pos);   // finishers' list lengths
    int* rowcnt = reinterpret_cast<int*>(pipe_smem + Ly.o_cnt);   // published list lengths

    for (int q = threadIdx.x; q < kDense * Wp; q += blockDim.x) dense[q] = -0.0;
    for (int q = threadIdx.x; q < Wp; q += blockDim.x) {
        dl[q] = q < W && q < n ? d0[q] : 0.0;
        lev[q] = 0;
        rowpos[q] = rowcnt[q] = 0;
    }
    if (threadIdx.x < kWalkers) s_ready[threadIdx.x] = -1;
    if (threadIdx.x == 0) {
        s_done = -1;
        s_stop = 0;
        s_result = 0;
        Lp[0] = 0;
    }
    __syncthreads();

    if (warp > 2 * kFin) {
        // ---- walker ----
        const int me = warp - 2 * kFin - 1;
        double* acc = accs + me * Wp;
        int slot = me % W;
        const int step = kWalkers % W;
        bool stop = false;
        for (int j = me; j < n && !stop; j += kWalkers) {
            int64_t p0 = Ap[j];
            const int64_t p1 = Ap[j + 1];
            // First entries of the column while the accumulator is in use.
            int64_t i0 = -1;
            double v0 = 0.0;
            if (p0 + lane < p1) {
                i0 = Ar[p0 + lane];
                v0 = Av[p0 + lane];
            }
            int at = 0;                  // nodes taken
            bool fresh = false;          // the accumulator holds A's column
            for (uint32_t spins = 0;; ++spins) {
                const int done_ = *(volatile int*)&s_done;
                const int cnt_ = *(volatile int*)&rowcnt[slot];
                const int done = __shfl_sync(all, done_, 0);
                int cnt = __shfl_sync(all, cnt_, 0);
                if (done == kPipeStop || spins >= limit) {
                    stop = true;
                    break;
                }
                // The accumulator is free once this walker's last column is
                // done, the slot is row j's once column j - W is.
                // Columns still to come before the list is complete: sleep for
                // most of them (polls take the finishers' issue slots).
                const int away = j - 1 - kLag - done;
                if (done < j - kWalkers || done < j - W) {
                    __nanosleep(200);
                    continue;
                }
                __threadfence_block();
                if (!fresh) {
                    for (int o = lane; o < W; o += 32) acc[o] = -0.0;
                    __syncwarp();
                    if (i0 > j && v0 != 0.0) acc[i0 - j] = v0;
                    for (int64_t k = p0 + 32 + lane; k < p1; k += 32) {
                        const int64_t i = Ar[k];
                        const double v = Av[k];
                        if (i > j && v != 0.0) acc[i - j] = v;
                    }
                    __syncwarp();
                    fresh = true;
                }
                if (at < cnt) {
                    const int2* row = list + slot * W;
                    for (int base = at; base < cnt; base += kBatch) {
                        // Entries of kBatch nodes in flight (an L2 round trip
                        // is ten times the work on one node).
                        int2 node[kBatch];
                        double f[kBatch], v[kBatch], v2[kBatch];
                        int i[kBatch], i2[kBatch];
#pragma unroll
                        for (int q = 0; q < kBatch; ++q)
                            node[q] = base + q < cnt ? row[base + q] : make_int2(0, 0);
#pragma unroll
                        for (int q = 0; q < kBatch; ++q) {
                            const int rest = node[q].y >> 16;
                            const double* Lg = Lv + node[q].x;
                            const uint16_t* Ig = offs + node[q].x;
                            f[q] = Lg[0];
                            v[q] = v2[q] = 0.0;
                            i[q] = i2[q] = 0;
                            if (lane < rest) {
                                v[q] = Lg[1 + lane];
                                i[q] = Ig[1 + lane];
                            }
                            if (rest > 32 && lane + 32 < rest) {
                                v2[q] = Lg[33 + lane];
                                i2[q] = Ig[33 + lane];
                            }
                        }
#pragma unroll
                        for (int q = 0; q < kBatch; ++q) {
                            const int rest = node[q].y >> 16;
                            double* from = acc - (node[q].y & 0xffff);   // offsets are from column k
                            if (lane < rest) {
                                double* x = from + i[q];
                                *x = (*x - v[q] * f[q]) + 0.0;
                            }
                            if (rest > 32 && lane + 32 < rest) {
                                double* x = from + i2[q];
                                *x = (*x - v2[q] * f[q]) + 0.0;
                            }
                            for (int c = 64 + lane; c < rest; c += 32) {
                                double* x = from + offs[node[q].x + 1 + c];
                                *x = (*x - Lv[node[q].x + 1 + c] * f[q]) + 0.0;
                            }
                            __syncwarp();
                        }
                    }
                    at = cnt;
                    spins = 0;
                }
                if (away <= 0) break;                 // the list was complete when read
                __nanosleep(away > 4 ? 1000 : away > 1 ? 200 : 40);
            }
            if (stop) break;
            __syncwarp();
            if (lane == 0) st_release(&s_ready[me], j);
            slot += step;
            if (slot >= W) slot -= W;
        }
    } else if (warp == kFin) {
        // ---- pivot: s_dj, s_sj, s_y of column j + 1 between the barriers of
        // column j, and the walker of column j + 2 ----
        int ready = 0;                        // columns below are known to be ready
        int wk = 0;
        auto await = [&](int c) {             // accumulator of column c, c = ready
            bool ok = false;
            for (uint32_t spins = 0; spins < limit; ++spins) {
                if (__shfl_sync(all, *(volatile int*)&s_ready[wk], 0) >= c) {
                    ok = true;
                    break;
                }
                __nanosleep(20);
            }
            __threadfence_block();
            if (!ok && lane == 0) {
                s_result = kIcholRetry;
                s_stop = 1;
            }
            ++ready;
            wk = wk + 1 == kWalkers ? 0 : wk + 1;
        };
        // y is one Newton step from rsqrt, which does not wait for the root:
        // rsqrt's 2^-51 squares to 2^-102.
        auto root = [&](double d) {
            const double s = sqrt(d);
            const double y0 = rsqrt(d);
            const double y = __fma_rn(__fma_rn(-s, y0, 1.0), y0, y0);
            if (lane == 0) {
                s_dj = d;
                s_sj = s;
                s_y = y;
            }
        };
        await(0);
        if (n > 1) await(1);
        root(dl[0]);
        pipe_barrier<kFin>(2);
        int slot = 1;
        for (int j = 0; j < n && !*(volatile int*)&s_stop; ++j) {
            pipe_barrier<kFin>(1);
            if (j + 1 < n) root(dl[slot]);
            if (lane == 0) st_release(&s_done, j - 1);     // it is in its rows' lists
            if (j + 2 < n) await(j + 2);
            pipe_barrier<kFin>(2);
            slot = slot + 1 == W ? 0 : slot + 1;
        }
        if (lane == 0) st_release(&s_done, kPipeStop);
    } else if (warp > kFin) {
        // ---- publishers: lane's offsets 1 + lane + 32 (me + kFin m) ----
        const int me = warp - kFin - 1;
        const bool first = me == 0 && lane == 0;
        int slot = 0;
        int64_t nnz = 0, nnz_at = 0;
        int look = look_cols > 0 ? look_cols : -1;      // column count of the next look
        double dnext = W < n ? d0[W] : 0.0;
        int psl[M], pcnt[M];                 // list lengths to publish for the column before
#pragma unroll
        for (int m = 0; m < M; ++m) pcnt[m] = 0;
        pipe_barrier<kFin>(2);
        for (int j = 0; j < n && !*(volatile int*)&s_stop; ++j) {
            // While the finishers make column j: lengths of the lists that
            // column j - 1 extended (written before the last barrier), and
            // what this column's rows hold.
            __threadfence_block();
            const double dj = s_dj, sj = s_sj;
            const int levj = lev[slot];
            int sl[M], lv[M], pos[M];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int o = 1 + lane + 32 * (me + kFin * m);
                if (pcnt[m]) *(volatile int*)&rowcnt[psl[m]] = pcnt[m];
                sl[m] = o >= W ? slot : slot + o >= W ? slot + o - W : slot + o;
                lv[m] = lev[sl[m]];
                pos[m] = rowpos[sl[m]];
            }
            pipe_barrier<kFin>(1);
            // Places in L: chunks in ascending offsets.
            const double* dc = dense + (j & (kDense - 1)) * Wp;
            double L[M];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int o = 1 + lane + 32 * (me + kFin * m);
                L[m] = o < W ? dc[o] : -0.0;
            }
            int before[M], total = 0;
#pragma unroll
            for (int c = 0; c < kFin * M; ++c) {
                if (c % kFin == me) before[c / kFin] = total & 0xffff;
                total += s_count[j & 1][c];
            }
            const int cn = total >> 16, kept = total & 0xffff;
            int64_t fail = 0;
            if (!(dj > 0.0)) fail = -1;                                              // ichol.py:80-81
            else if (nnz + 1 + cn > max_nnz || nnz + 1 + cn > cap) fail = -2;        // ichol.py:82-83
            if (fail) {
                if (first) {
                    s_result = fail;
                    s_stop = 1;
                }
            } else {
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    pcnt[m] = 0;
                    const bool keep = has_entry(L[m]);
                    const unsigned km = __ballot_sync(all, keep);
                    if (keep) {
                        const int o = 1 + lane + 32 * (me + kFin * m);
                        const int r = before[m] + __popc(km & lt);
                        const int64_t g = nnz + 1 + r;
                        Lv[g] = L[m];
                        Lr[g] = j + o;
                        offs[g] = (uint16_t)o;
                        if (lv[m] <= levj) lev[sl[m]] = levj + 1;
                        if (o > kLag) {
                            const int p = pos[m];
                            rowpos[sl[m]] = p + 1;
                            list[sl[m] * W + p] = make_int2((int)g, (kept - 1 - r) << 16 | o);
                            psl[m] = sl[m];
                            pcnt[m] = p + 1;
                        }
                    }
                }
                if (first) {
                    Lv[nnz] = sj;
                    Lr[nnz] = j;
                    Lp[j + 1] = nnz + 1 + kept;
                    level[j] = levj;
                    // The slot's next row.
                    dl[slot] = dnext;
                    lev[slot] = 0;
                    rowpos[slot] = 0;
                    *(volatile int*)&rowcnt[slot] = 0;
                    if (j + 1 + W < n) dnext = d0[j + 1 + W];
                }
                nnz += 1 + kept;
                slot = slot + 1 == W ? 0 : slot + 1;
                if (j + 1 == look) {
                    if (look > look_cols && nnz - nnz_at > dense_nnz && first) {
                        s_result = kIcholDense;
                        s_stop = 1;
                    }
                    nnz_at = nnz;
                    look = look + look_cols <= look_end ? look + look_cols : -1;
                }
            }
            pipe_barrier<kFin>(2);
        }
        if (first && !s_result) s_result = nnz;
    } else {
        // ---- finishers: lane's offsets 1 + lane + 32 (warp + kFin m) ----
        int slot = 0, wk = 0;
        double rnow = rsum[0], rnext = n > 1 ? rsum[1] : 0.0;
        double a[M];
        // The accumulator of column c and the terms of the dense columns.
        auto gather = [&](int c) {
            const double* acc = accs + wk * Wp;
            wk = wk + 1 == kWalkers ? 0 : wk + 1;
            double f[kLag], x[kLag][M];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int o = 1 + lane + 32 * (warp + kFin * m);
                a[m] = o < W ? acc[o] : -0.0;
            }
#pragma unroll
            for (int b = kLag; b >= 1; --b) {
                const double* dc = dense + ((c - b) & (kDense - 1)) * Wp;
                f[b - 1] = dc[b];
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const int o = 1 + lane + 32 * (warp + kFin * m);
                    x[b - 1][m] = o < W ? dc[o + b] : -0.0;
                }
            }
#pragma unroll
            for (int b = kLag; b >= 1; --b) {
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const double t = (a[m] - x[b - 1][m] * f[b - 1]) + 0.0;
                    if (has_entry(f[b - 1]) && has_entry(x[b - 1][m])) a[m] = t;
                }
            }
        };
        pipe_barrier<kFin>(2);
        if (!*(volatile int*)&s_stop) gather(0);
        for (int j = 0; j < n && !*(volatile int*)&s_stop; ++j) {
            // Quotients, thresholds, diagonal updates, dense copy.
            const double sj = s_sj, y = s_y;
            const double rel = rel_discard * rnow;
            rnow = rnext;
            if (j + 2 < n) rnext = rsum[j + 2];
            double L[M], du[M];
            int sl[M];
            bool odd = !root_range(sj);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int o = 1 + lane + 32 * (warp + kFin * m);
                sl[m] = o >= W ? slot : slot + o >= W ? slot + o - W : slot + o;
                du[m] = dl[sl[m]];
                odd |= has_entry(a[m]) && !(a[m] == 0.0 || mid_range(a[m]));
                L[m] = pipe_quotient(a[m], sj, y);
            }
            if (__any_sync(all, odd)) {
                // + 0.0: a quotient that underflows to -0.0 is an entry too
                // (kept where the threshold is negative).
#pragma unroll
                for (int m = 0; m < M; ++m) L[m] = a[m] / sj + 0.0;
            }
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int o = 1 + lane + 32 * (warp + kFin * m);
                const bool in = has_entry(a[m]);
                const bool keep = in && fabs(L[m]) > discard && fabs(a[m]) > rel;
                if (in && (diag_keep || keep)) dl[sl[m]] = du[m] - L[m] * L[m];
                if (o < W) dense[(j & (kDense - 1)) * Wp + o] = keep ? L[m] : -0.0;
                const unsigned fm = __ballot_sync(all, in);
                const unsigned km = __ballot_sync(all, keep);
                if (lane == 0) s_count[j & 1][warp + kFin * m] = __popc(fm) << 16 | __popc(km);
            }
            pipe_barrier<kFin>(1);
            slot = slot + 1 == W ? 0 : slot + 1;
            if (j + 1 < n) gather(j + 1);
            pipe_barrier<kFin>(2);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) *result = s_result;
}

// Level histogram / order of rows, and the row (CSR) view of L used by the
// forward solve. All small single-purpose kernels.
__global__ void k_level_count(int64_t n, const int* __restrict__ level, int64_t* cnt,
                              int* maxlevel) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    atomicAdd((unsigned long long*)&cnt[level[i]], 1ull);
    atomicMax(maxlevel, level[i]);
}

__global__ void k_level_scatter(int64_t n, const int* __restrict__ level, int64_t* fill,
                                int* order) {
    // Sequential within one thread per level bucket would be slow; rows are
    // placed with atomics, then each level segment is sorted by row.
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long at = atomicAdd((unsigned long long*)&fill[level[i]], 1ull);
    order[at] = (int)i;
}

// Insertion-sort each level segment so the schedule is deterministic.
__global__ void k_level_sort(const int64_t* __restrict__ lptr, int nlevels, int* order) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nlevels) return;
    const int64_t a = lptr[l], b = lptr[l + 1];
    for (int64_t k = a + 1; k < b; ++k) {
        const int v = order[k];
        int64_t q = k - 1;
        while (q >= a && order[q] > v) {
            order[q + 1] = order[q];
            --q;
        }
        order[q + 1] = v;
    }
}

__global__ void k_row_count(int64_t n, const int64_t* __restrict__ Lp, const int64_t* __restrict__ Lr,
                            int64_t* rcnt) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    for (int64_t k = Lp[j] + 1; k < Lp[j + 1]; ++k)
        atomicAdd((unsigned long long*)&rcnt[Lr[k]], 1ull);
}

// Row view entries in ascending column order: column j writes its entry
// of row i at the slot given by the number of columns < j with an entry in
// row i — computed by walking columns in order within one thread per row
// would be quadratic, so entries are appended with atomics and each row is
// sorted afterwards.
__global__ void k_row_fill(int64_t n, const int64_t* __restrict__ Lp, const int64_t* __restrict__ Lr,
                           const double* __restrict__ Lv, int64_t* rfill, int64_t* Rc, double* Rv) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    for (int64_t k = Lp[j] + 1; k < Lp[j + 1]; ++k) {
        const int64_t i = Lr[k];
        const unsigned long long at = atomicAdd((unsigned long long*)&rfill[i], 1ull);
        Rc[at] = j;
        Rv[at] = Lv[k];
    }
}

// Rows of up to kRowSortMax entries: one warp per row, entries in registers
// (8 a lane); each entry's place is the number of smaller column indices in
// its row (the indices of a row are distinct), counted by broadcasting every
// key through the warp.
constexpr int kRowSortMax = 256;

__global__ void k_row_sort_warp(int64_t n, const int64_t* __restrict__ Rp, int64_t* Rc, double* Rv) {
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= n) return;
    const int64_t b = Rp[i];
    const int64_t len = Rp[i + 1] - b;
    if (len <= 1 || len > kRowSortMax) return;
    int64_t c[8];
    double v[8];
    int rank[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int k = lane + 32 * u;
        c[u] = k < len ? Rc[b + k] : INT64_MAX;
        v[u] = k < len ? Rv[b + k] : 0.0;
        rank[u] = 0;
    }
    const int U = (int)((len + 31) >> 5);
#pragma unroll
    for (int u2 = 0; u2 < 8; ++u2) {
        if (u2 < U) {
            for (int src = 0; src < 32; ++src) {
                const int64_t key = __shfl_sync(0xffffffffu, c[u2], src);
#pragma unroll
                for (int u = 0; u < 8; ++u) rank[u] += key < c[u] ? 1 : 0;
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int k = lane + 32 * u;
        if (k < len) {
            Rc[b + rank[u]] = c[u];
            Rv[b + rank[u]] = v[u];
        }
    }
}

// Longer rows: insertion sort by one thread.
__global__ void k_row_sort(int64_t n, const int64_t* __restrict__ Rp, int64_t* Rc, double* Rv) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (Rp[i + 1] - Rp[i] <= kRowSortMax) return;
    for (int64_t k = Rp[i] + 1; k < Rp[i + 1]; ++k) {
        const int64_t c = Rc[k];
        const double v = Rv[k];
        int64_t q = k - 1;
        while (q >= Rp[i] && Rc[q] > c) {
            Rc[q + 1] = Rc[q];
            Rv[q + 1] = Rv[q];
            --q;
        }
        Rc[q + 1] = c;
        Rv[q + 1] = v;
    }
}

// x = L^-T L^-1 b. Forward: y_i = (b_i - sum_{j<i} L_ij y_j) / L_ii with
// the subtractions in ascending j (the column sweep of
// _backsub_L_csc_inplace applies them in that order); backward: x_i =
// (y_i - sum_{k>i} L_ki x_k) / L_ii over column i in ascending k
// (_backsub_LT_csc_inplace). Levels run forward, then in reverse.
__global__ void __launch_bounds__(kIcholThreads)
k_ichol_solve(int64_t n, int nlevels, const int64_t* __restrict__ lptr, const int* __restrict__ order,
              const int64_t* __restrict__ Lp, const int64_t* __restrict__ Lr,
              const double* __restrict__ Lv, const int64_t* __restrict__ Rp,
              const int64_t* __restrict__ Rc, const double* __restrict__ Rv,
              const double* __restrict__ b, double* x, const InstState* st) {
    if (st && st->status != kRunning) return;
    for (int l = 0; l < nlevels; ++l) {
        for (int64_t q = lptr[l] + threadIdx.x; q < lptr[l + 1]; q += blockDim.x) {
            const int64_t i = order[q];
            double s = b[i];
            for (int64_t k = Rp[i]; k < Rp[i + 1]; ++k) s -= Rv[k] * x[Rc[k]];
            x[i] = s / Lv[Lp[i]];
        }
        __syncthreads();
    }
    for (int l = nlevels - 1; l >= 0; --l) {
        for (int64_t q = lptr[l] + threadIdx.x; q < lptr[l + 1]; q += blockDim.x) {
            const int64_t i = order[q];
            double s = x[i];
            for (int64_t k = Lp[i] + 1; k < Lp[i + 1]; ++k) s -= Lv[k] * x[Lr[k]];
            x[i] = s / Lv[Lp[i]];
        }
        __syncthreads();
    }
}

// The same solves with x in shared memory (n <= kIcholSmemRows) and one warp
// per row: the lanes split the row's dot product (so the subtractions of a
// row are summed in a different order than the reference, a difference of
// rounding only) and each warp loads the index/value data of its first row
// of the next level before the level barrier, so a level costs one shared-
// memory gather, a warp reduction and a barrier.
struct RowPrefetch {
    int64_t i, k0, k1;
    int64_t c;     // first entry of this lane (column / row index)
    double v;
};

template <bool FWD>
__device__ __forceinline__ RowPrefetch prefetch_row(int64_t q, int64_t qend, const int* order,
                                                    const int64_t* Xp, const int64_t* Xi,
                                                    const double* Xv, int lane) {
    RowPrefetch r{-1, 0, 0, 0, 0.0};
    if (q < qend) {
        r.i = order[q];
        r.k0 = Xp[r.i] + (FWD ? 0 : 1);
        r.k1 = Xp[r.i + 1];
        const int64_t k = r.k0 + lane;
        if (k < r.k1) {
            r.c = Xi[k];
            r.v = Xv[k];
        }
    }
    return r;
}

template <bool FWD>
__device__ __forceinline__ void solve_sweep(int nlevels, const int64_t* __restrict__ lptr,
                                            const int* __restrict__ order,
                                            const int64_t* __restrict__ Xp,
                                            const int64_t* __restrict__ Xi,
                                            const double* __restrict__ Xv,
                                            const int64_t* __restrict__ Lp,
                                            const double* __restrict__ Lv, double* sx) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int l = FWD ? 0 : nlevels - 1;
    RowPrefetch pf = prefetch_row<FWD>(lptr[l] + warp, lptr[l + 1], order, Xp, Xi, Xv, lane);
    for (int step = 0; step < nlevels; ++step, l += FWD ? 1 : -1) {
        const int64_t qend = lptr[l + 1];
        int64_t q = lptr[l] + warp;
        RowPrefetch cur = pf;
        // Prefetch this warp's first row of the next level (its data does
        // not depend on x).
        if (step + 1 < nlevels) {
            const int ln = FWD ? l + 1 : l - 1;
            pf = prefetch_row<FWD>(lptr[ln] + warp, lptr[ln + 1], order, Xp, Xi, Xv, lane);
        }
        while (cur.i >= 0) {
            double acc = (cur.k0 + lane < cur.k1) ? cur.v * sx[cur.c] : 0.0;
            for (int64_t k = cur.k0 + 32 + lane; k < cur.k1; k += 32) acc += Xv[k] * sx[Xi[k]];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) sx[cur.i] = (sx[cur.i] - acc) / Lv[Lp[cur.i]];
            q += nw;
            cur = prefetch_row<FWD>(q, qend, order, Xp, Xi, Xv, lane);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kIcholThreads)
k_ichol_solve_smem(int64_t n, int nlevels, const int64_t* __restrict__ lptr,
                   const int* __restrict__ order, const int64_t* __restrict__ Lp,
                   const int64_t* __restrict__ Lr, const double* __restrict__ Lv,
                   const int64_t* __restrict__ Rp, const int64_t* __restrict__ Rc,
                   const double* __restrict__ Rv, const double* __restrict__ b, double* x,
                   const InstState* st) {
    extern __shared__ double s_x[];
    if (st && st->status != kRunning) return;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s_x[i] = b[i];
    __syncthreads();
    if (nlevels > 0) {
        solve_sweep<true>(nlevels, lptr, order, Rp, Rc, Rv, Lp, Lv, s_x);
        solve_sweep<false>(nlevels, lptr, order, Lp, Lr, Lv, Lp, Lv, s_x);
    }
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) x[i] = s_x[i];
}

// ---------------------------------------------------------------------------
// Streamed level-scheduled solves (n <= kStreamMaxRows). Both sweeps run in
// one CTA with x in shared memory. The rows of each sweep, in level order,
// are packed at factorisation time into chunks (one level, or a part of a
// level, of at most kStreamRowsMax rows and kStreamEntsMax entries), each a
// contiguous 16-byte-aligned block:
//
//   StreamHead   own row and entry counts, and the offset / size of the
//                block kStreamStages chunks later (the next one to fetch
//                into this stage)
//   StreamRow[rows]   row index, first entry, entry count, diagonal
//   double[ents]      L values of the row terms
//   int[ents]         their x indices       (ents padded to a multiple of 4)
//
// A warp of its own keeps kStreamStages chunks in flight with bulk copies into
// a shared-memory ring (completion on one mbarrier per stage) and waits for
// each chunk two steps before it is used, so the other warps see its data
// through the block barrier that ends a step. They take the record and the
// entries of their row of the next chunk into registers while this one's sums
// are made (neither depends on x); what is left on the chain from level to
// level is the gather of x, the warp's reduction, the quotient (a corrected
// product with the reciprocal that the packing made, rounded as the division)
// and the barrier. Within a row the terms are summed lane-strided and reduced
// across the warp, as in k_ichol_solve_smem, and x_i = (x_i - sum) / L_ii as
// the reference's back substitutions (ichol.py:116-145). 7,815 rows in 2,301
// levels: 1.48 -> 1.21 ms for both sweeps, about 500 cycles per chunk, of
// which the five shuffle steps of the reduction are the largest part. Terms
// beyond the 64 in registers go in groups whose loads are in flight together:
// 7,200 rows of 289 entries 10.3 (two at a time, no registers) and 14.0 (one
// at a time) -> 8.9 ms, 10,985 rows of 45 entries 3.01 -> 2.42 ms.
// ---------------------------------------------------------------------------

constexpr int kStreamWarps = 8;       // that take rows; one more for the copies
constexpr int kStreamThreads = 32 * (kStreamWarps + 1);
constexpr size_t kStreamStageBytes =
    sizeof(StreamHead) + kStreamRowsMax * sizeof(StreamRow) + kStreamEntsMax * 12;
static_assert(kStreamStageBytes % 16 == 0, "stages are 16-byte aligned");

size_t ichol_stream_smem(int64_t n) {
    return kStreamStages * kStreamStageBytes + (size_t)n * sizeof(double);
}

// x_i from its numerator: the division where the record does not vouch for the
// reciprocal, or the numerator is outside the quotient's range.
__device__ __forceinline__ double stream_quotient(double num, const StreamRow& rw) {
    if (rw.fast && (num == 0.0 || mid_range(num))) return pipe_quotient(num, rw.diag, rw.inv);
    return num / rw.diag;
}

__global__ void __launch_bounds__(kStreamThreads)
k_ichol_solve_stream(int64_t n, int total, StreamFirst first, const unsigned char* __restrict__ blob,
                     const double* __restrict__ b, double* x, const InstState* st, uint32_t limit) {
    extern __shared__ __align__(16) unsigned char ss_smem[];
    __shared__ uint64_t full[kStreamStages];
    __shared__ int s_bad[2];      // by step parity: written in a step, read in the next
    if (st && st->status != kRunning) return;
    double* sx = reinterpret_cast<double*>(ss_smem + kStreamStages * kStreamStageBytes);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool copier = warp == kStreamWarps && lane == 0;
    auto landed = [&](int c) {
        return c >= total ||
               mbar_wait(&full[c % kStreamStages], (uint32_t)(c / kStreamStages) & 1u, limit);
    };
    if (copier) {
        for (int q = 0; q < kStreamStages; ++q) mbar_init(&full[q], 1);
        for (int q = 0; q < kStreamStages && q < total; ++q) {
            if (first.bytes[q] <= 0) continue;
            mbar_expect_tx(&full[q], (uint32_t)first.bytes[q]);
            bulk_load(ss_smem + q * kStreamStageBytes, blob + first.off[q], (uint32_t)first.bytes[q],
                      &full[q]);
        }
        s_bad[1] = !(landed(0) && landed(1));
    }
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) sx[i] = b[i];
    __syncthreads();
    // Row of this warp in the coming chunk.
    StreamRow rw;
    double v0 = 0.0, v1 = 0.0;
    int c0 = 0, c1 = 0;
    bool mine = false;
    auto chunk = [&](int c, const StreamRow*& rec, const double*& val, const int*& col) {
        const unsigned char* stage = ss_smem + (c % kStreamStages) * kStreamStageBytes;
        const StreamHead* h = reinterpret_cast<const StreamHead*>(stage);
        rec = reinterpret_cast<const StreamRow*>(stage + sizeof(StreamHead));
        val = reinterpret_cast<const double*>(stage + sizeof(StreamHead) + h->rows * sizeof(StreamRow));
        col = reinterpret_cast<const int*>(val + h->ents);
        return h->rows;
    };
    // Terms e, e + 32, ... of a row, the loads of kTerms in flight.
    auto terms = [&](const double* val, const int* col, int count, int e, double& acc) {
        constexpr int kTerms = 4;
        for (; e < count; e += 32 * kTerms) {
            double v[kTerms];
            int i[kTerms];
#pragma unroll
            for (int u = 0; u < kTerms; ++u) {
                v[u] = 0.0;
                i[u] = 0;
                if (e + 32 * u < count) {
                    v[u] = val[e + 32 * u];
                    i[u] = col[e + 32 * u];
                }
            }
            double x[kTerms];
#pragma unroll
            for (int u = 0; u < kTerms; ++u) x[u] = sx[i[u]];
#pragma unroll
            for (int u = 0; u < kTerms; ++u)
                if (e + 32 * u < count) acc += v[u] * x[u];
        }
    };
    auto fetch = [&](int c) {
        const StreamRow* rec;
        const double* val;
        const int* col;
        mine = c < total && warp < chunk(c, rec, val, col);
        if (!mine) return;
        rw = rec[warp];
        v0 = v1 = 0.0;
        c0 = c1 = rw.row;
        if (lane < rw.count) {
            v0 = val[rw.start + lane];
            c0 = col[rw.start + lane];
        }
        if (lane + 32 < rw.count) {
            v1 = val[rw.start + lane + 32];
            c1 = col[rw.start + lane + 32];
        }
    };
    int c = 0;
    int64_t next_off = 0;
    int next_bytes = 0, issued = min(total, kStreamStages);
    bool bad = s_bad[1] != 0;
    if (warp < kStreamWarps && !bad) fetch(0);
    for (; c < total && !bad; ++c) {
        if (warp < kStreamWarps) {
            const bool have = mine;
            const StreamRow r = rw;
            double acc = 0.0, x0 = 0.0, x1 = 0.0, xr = 0.0, w0 = v0, w1 = v1;
            const bool two = have && lane + 32 < r.count;
            if (have) {
                x0 = sx[c0];
                x1 = sx[c1];
                xr = sx[r.row];
            }
            fetch(c + 1);
            const StreamRow* rec;
            const double* val;
            const int* col;
            const int rows = chunk(c, rec, val, col);
            if (have) {
                if (lane < r.count) acc += w0 * x0;
                if (two) acc += w1 * x1;
                if (r.count > 64) terms(val + r.start, col + r.start, r.count, lane + 64, acc);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                if (lane == 0) sx[r.row] = stream_quotient(xr - acc, r);
            }
            for (int k = warp + kStreamWarps; k < rows; k += kStreamWarps) {
                const StreamRow rk = rec[k];
                acc = 0.0;
                terms(val + rk.start, col + rk.start, rk.count, lane, acc);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                if (lane == 0) sx[rk.row] = stream_quotient(sx[rk.row] - acc, rk);
            }
        } else if (copier) {
            // The stage that the last step left, then the chunk of the step
            // after the next.
            if (next_bytes > 0) {
                uint64_t* bar = &full[(c - 1) % kStreamStages];
                fence_proxy_async();
                mbar_expect_tx(bar, (uint32_t)next_bytes);
                bulk_load(ss_smem + ((c - 1) % kStreamStages) * kStreamStageBytes, blob + next_off,
                          (uint32_t)next_bytes, bar);
                ++issued;
            }
            const StreamHead* h =
                reinterpret_cast<const StreamHead*>(ss_smem + (c % kStreamStages) * kStreamStageBytes);
            next_off = h->next_off;
            next_bytes = h->next_bytes;
            s_bad[c & 1] = !landed(c + 2);
        }
        __syncthreads();          // level barrier; the stage is free again
        bad = s_bad[c & 1] != 0;
    }
    if (bad) {
        // A copy did not complete: the result is NaN, and copies still in
        // flight are waited for (bounded) before the CTA leaves.
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) x[i] = __longlong_as_double(0x7ff8000000000000ll);
        if (copier) {
            for (int k = c; k < issued; ++k) landed(k);
        }
        __syncthreads();
        return;
    }
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) x[i] = sx[i];
}

// Pack the chunk blocks of both sweeps. One warp per row record: its entries
// (x indices narrowed to int) and its record; one thread per chunk writes the
// head and zeroes the entry padding.
__global__ void k_stream_pack_rows(int nrec, const StreamPackRow* __restrict__ recs,
                                   const int64_t* __restrict__ Rc, const double* __restrict__ Rv,
                                   const int64_t* __restrict__ Lr, const double* __restrict__ Lv,
                                   const int64_t* __restrict__ Lp, unsigned char* blob) {
    const int w = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= nrec) return;
    const StreamPackRow R = recs[w];
    unsigned char* chunk = blob + R.chunk_off;
    StreamRow* rec = reinterpret_cast<StreamRow*>(chunk + sizeof(StreamHead)) + R.slot;
    double* val = reinterpret_cast<double*>(chunk + sizeof(StreamHead) + R.rows * sizeof(StreamRow));
    int* col = reinterpret_cast<int*>(val + R.ents);
    const int64_t* ci = R.backward ? Lr : Rc;
    const double* cv = R.backward ? Lv : Rv;
    for (int e = lane; e < R.count; e += 32) {
        val[R.start + e] = cv[R.src + e];
        col[R.start + e] = (int)ci[R.src + e];
    }
    if (lane == 0) {
        StreamRow rw;
        rw.row = R.row;
        rw.start = R.start;
        rw.count = R.count;
        rw.diag = Lv[Lp[R.row]];
        rw.inv = 1.0 / rw.diag;
        rw.fast = root_range(rw.diag);
        *rec = rw;
    }
}

__global__ void k_stream_pack_heads(int nchunks, const StreamPackChunk* __restrict__ ch,
                                    unsigned char* blob) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nchunks) return;
    const StreamPackChunk C = ch[c];
    StreamHead h;
    h.next_off = c + kStreamStages < nchunks ? ch[c + kStreamStages].off : 0;
    h.next_bytes = c + kStreamStages < nchunks ? ch[c + kStreamStages].bytes : 0;
    h.rows = C.rows;
    h.ents = C.ents;
    h.pad[0] = h.pad[1] = h.pad[2] = 0;
    *reinterpret_cast<StreamHead*>(blob + C.off) = h;
    double* val = reinterpret_cast<double*>(blob + C.off + sizeof(StreamHead) + C.rows * sizeof(StreamRow));
    int* col = reinterpret_cast<int*>(val + C.ents);
    for (int e = C.used; e < C.ents; ++e) {
        val[e] = 0.0;
        col[e] = 0;
    }
}

void ichol_launch_stream_pack(int nrec, const StreamPackRow* recs, int nchunks,
                              const StreamPackChunk* chunks, const int64_t* Rc, const double* Rv,
                              const int64_t* Lr, const double* Lv, const int64_t* Lp,
                              unsigned char* blob, cudaStream_t s) {
    if (nrec > 0)
        k_stream_pack_rows<<<(unsigned)((nrec * 32 + 255) / 256), 256, 0, s>>>(nrec, recs, Rc, Rv, Lr,
                                                                               Lv, Lp, blob);
    if (nchunks > 0)
        k_stream_pack_heads<<<(unsigned)((nchunks + 127) / 128), 128, 0, s>>>(nchunks, chunks, blob);
}

void ichol_launch_solve_stream(int64_t n, int total, const StreamFirst& first,
                               const unsigned char* blob, const double* b, double* x,
                               const InstState* st, uint32_t limit, cudaStream_t s) {
    k_ichol_solve_stream<<<1, kStreamThreads, ichol_stream_smem(n), s>>>(n, total, first, blob, b, x,
                                                                         st, limit);
}

// The forward sweep above overwrites x in place: y lives in x. For the
// forward pass to read y_j of earlier levels and b_i of its own row, b and
// x may alias (the reference also works in place on a copy of b).

void ichol_launch_init(int64_t n, const int64_t* Ap, const int64_t* Ar, const double* Av,
                       double shift, double* d, double* rsum, int* level, unsigned long long* band,
                       cudaStream_t s) {
    if (n > 0) k_ichol_init<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, Ap, Ar, Av, shift, d, rsum, level, band);
}

// The pipelined kernel, for the bandwidths that its shared memory takes; limit:
// polls after which a wait gives up; look_cols > 0: ends with kIcholDense if the
// second look_cols columns, or any of the next up to column look_end, kept more
// than dense_nnz entries. False: not launched. `list` holds max(W, kPipeMinW)^2 doubles.
bool ichol_launch_factor_pipe(int64_t n, int64_t W, const int64_t* Ap, const int64_t* Ar,
                              const double* Av, const double* d, const double* rsum, int* level,
                              int64_t* Lp, int64_t* Lr, double* Lv, double* list, uint16_t* offs, int64_t cap,
                              double discard, int64_t max_nnz, double rel, int diag_keep,
                              int64_t* result, uint32_t limit, int look_cols, int64_t look_end,
                              int64_t dense_nnz, cudaStream_t s) {
    W = W < kPipeMinW ? kPipeMinW : W;
    if (W > 32 * kPipeMaxChunks + 1 || n > kPipeMax || cap > kPipeMax) return false;
    const int chunks = (int)((W - 1 + 31) / 32);
    const int fin = chunks <= 8 ? 4 : chunks <= 12 ? 6 : 8;
    const PipeLayout L = pipe_layout(W, pipe_walkers(fin));
    if (L.bytes > kFactorSmem - 512) return false;
    auto kern = chunks <= 4 ? k_ichol_factor_pipe<4, 1>
              : chunks <= 8 ? k_ichol_factor_pipe<4, 2>
              : chunks <= 12 ? k_ichol_factor_pipe<6, 2>
              : chunks <= 16 ? k_ichol_factor_pipe<8, 2> : k_ichol_factor_pipe<8, 4>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.bytes) !=
        cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    kern<<<1, 32 * pipe_warps(fin), L.bytes, s>>>((int)n, (int)W, Ap, Ar, Av, d, rsum, level, Lp, Lr, Lv,
                                          reinterpret_cast<int2*>(list), offs, cap, discard, max_nnz, rel,
                                          diag_keep, result, limit, look_cols, (int)look_end, dense_nnz);
    return true;
}

void ichol_launch_factor(int64_t n, int64_t W, const int64_t* Ap, const int64_t* Ar,
                         const double* Av, double* d, const double* rsum, int* level, double* F,
                         uint8_t* pat, int* cand, double* keptv, int64_t* kepti, int64_t* Lp,
                         int64_t* Lr, double* Lv, int64_t cap, double discard, int64_t max_nnz,
                         double rel_discard, int diag_keep, int64_t* result, cudaStream_t s) {
    k_ichol_factor<<<1, kIcholThreads, 0, s>>>(n, W, Ap, Ar, Av, d, rsum, level, F, pat, cand, keptv,
                                               kepti, Lp, Lr, Lv, cap, discard, max_nnz, rel_discard,
                                               diag_keep, result);
}

void ichol_launch_levels(int64_t n, const int* level, int64_t* cnt, int* maxlevel, cudaStream_t s) {
    if (n > 0) k_level_count<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, level, cnt, maxlevel);
}

void ichol_launch_level_scatter(int64_t n, const int* level, int64_t* fill, int* order,
                                const int64_t* lptr, int nlevels, cudaStream_t s) {
    if (n > 0) k_level_scatter<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, level, fill, order);
    if (nlevels > 0) k_level_sort<<<(nlevels + 127) / 128, 128, 0, s>>>(lptr, nlevels, order);
}

void ichol_launch_rows(int64_t n, const int64_t* Lp, const int64_t* Lr, const double* Lv,
                       int64_t* rcnt, cudaStream_t s) {
    if (n > 0) k_row_count<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, Lp, Lr, rcnt);
}

void ichol_launch_row_fill(int64_t n, const int64_t* Lp, const int64_t* Lr, const double* Lv,
                           int64_t* rfill, int64_t* Rc, double* Rv, const int64_t* Rp,
                           cudaStream_t s) {
    if (n > 0) {
        k_row_fill<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, Lp, Lr, Lv, rfill, Rc, Rv);
        k_row_sort_warp<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(n, Rp, Rc, Rv);
        k_row_sort<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, Rp, Rc, Rv);
    }
}

// Raise the shared-memory limit of the shared-memory solve; called when a
// factor is built, before any solve can be captured.
void ichol_prepare() {
    cudaFuncSetAttribute(k_ichol_solve_smem, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(kIcholSmemRows * sizeof(double)));
    cudaFuncSetAttribute(k_ichol_solve_stream, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)ichol_stream_smem(kStreamMaxRows));
}

void ichol_launch_solve(int64_t n, int nlevels, const int64_t* lptr, const int* order,
                        const int64_t* Lp, const int64_t* Lr, const double* Lv, const int64_t* Rp,
                        const int64_t* Rc, const double* Rv, const double* b, double* x,
                        const InstState* st, cudaStream_t s) {
    if (n <= kIcholSmemRows) {
        k_ichol_solve_smem<<<1, kIcholThreads, n * sizeof(double), s>>>(
            n, nlevels, lptr, order, Lp, Lr, Lv, Rp, Rc, Rv, b, x, st);
        return;
    }
    k_ichol_solve<<<1, kIcholThreads, 0, s>>>(n, nlevels, lptr, order, Lp, Lr, Lv, Rp, Rc, Rv, b, x, st);
}

}  // namespace pmb
