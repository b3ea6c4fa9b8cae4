// Thresholded incomplete Cholesky with the band front on chip, for bands whose
// columns keep many entries.
//
// A cluster of C CTAs keeps the W x W front of k_ichol_factor (ichol.cu) in
// distributed shared memory, CTA r owning the slots s with
// s mod C = r (at most S = ceil(W / C) of them) with their FP64 values,
// pattern bytes, ring entries of the diagonal d and of the dependency level.
// Per column j:
//
//   phase F  warp 0 of EVERY CTA reads slot j from its owner (one DSMEM round
//            trip) and runs the serial part of the column (pivot, threshold,
//            compaction) on identical data with identical instructions, so all
//            CTAs hold the same kept list and take the same control path; the
//            owner writes the column of L. Meanwhile the last warp recycles the
//            slot of column j - 1 for column j - 1 + W from registers it loaded
//            one column earlier (A's entries) and two columns earlier (A's
//            column pointers), so no global load latency is on the chain.
//   phase P  each CTA applies the pair updates F[ib][ia - ib] -= L_ia L_ib whose
//            target column ib it owns, and the diagonal and level updates of
//            the rows it owns: every write is CTA-local.
//
// One cluster barrier per column orders phase P of column j before phase F of
// column j + 1 in every CTA. Updates land in the same order as in
// k_ichol_factor (column order, one pair per front entry per column), so the
// two kernels produce identical factors.
//
// A column's m (m - 1) / 2 updates are spread over C SMs, where the pipeline of
// ichol.cu has one: bound by the cluster barrier and the column's phase F while
// columns are short (2.3 us a column with 34 entries kept of W = 301, the
// pipeline 0.9), by the updates of the busiest CTA when they are long. The two
// cross where m C is about 900 (us a column, pipeline / cluster):
//   W = 271, C = 4   m 147: 4.5 / 5.3   199: 7.4 / 7.5   267: 11.5 / 10.8
//   W = 351, C = 6   m 130: 3.6 / 4.2   153: 4.9 / 4.9   346: 17.8 / 11.9
//   W = 401, C = 7   m 107: 3.3 / 3.7   132: 4.5 / 4.2   395: 24.4 / 13.3
#include <cooperative_groups.h>

#include "pm_common.cuh"
#include "ichol.cuh"

namespace pmb {

constexpr int kClThreads = 512;
constexpr int kClMaxChunks = 14;      // offsets 1 .. W - 1 in chunks of 32: W <= 449
constexpr int kClMaxCluster = 8;      // portable cluster size
constexpr size_t kClSmemLimit = 227 * 1024 - 256;

struct ClLayout {
    int64_t Wp, S;
    size_t o_F, o_d, o_kv, o_cL, o_lev, o_ki, o_ci, o_own, o_pre, o_pat, bytes;
};

__host__ __device__ inline ClLayout cl_layout(int64_t W, int C) {
    ClLayout L;
    L.Wp = (W + 7) & ~(int64_t)7;
    L.S = (W + C - 1) / C;
    size_t o = 0;
    L.o_F = o;   o += (size_t)(L.S * L.Wp) * sizeof(double);
    L.o_d = o;   o += (size_t)L.S * sizeof(double);
    L.o_kv = o;  o += (size_t)W * sizeof(double);
    L.o_cL = o;  o += (size_t)W * sizeof(double);
    L.o_lev = o; o += (size_t)L.S * sizeof(int);
    L.o_ki = o;  o += (size_t)W * sizeof(int);
    L.o_ci = o;  o += (size_t)W * sizeof(int);
    L.o_own = o; o += (size_t)W * sizeof(int);
    L.o_pre = o; o += (size_t)W * sizeof(int);
    L.o_pat = o; o += (size_t)(L.S * L.Wp);
    L.bytes = (o + 15) & ~(size_t)15;
    return L;
}

// Smallest cluster size whose per-CTA share of the front fits in shared
// memory; 0 when none up to the portable limit does (or W is too wide for
// the register chunks of phase F).
int ichol_cluster_size(int64_t W) {
    if (W < 1 || W - 1 > 32 * kClMaxChunks) return 0;
    for (int C = 1; C <= kClMaxCluster; ++C)
        if (cl_layout(W, C).bytes <= kClSmemLimit) return C;
    return 0;
}

// NCH: 32-offset chunks of a front column held in registers by phase F
// (ceil((W - 1) / 32) rounded up to 2, 4, 8 or 14). Slots are tracked
// incrementally in 32-bit arithmetic. Phase F compacts the column's
// candidates first and divides only those, lane-strided: an FP64 division
// costs about 130 cycles of latency (about 300 with a zero numerator), and
// a column has a quarter of its offsets as candidates or fewer.
template <int NCH>
__global__ void __launch_bounds__(kClThreads, 1)
k_ichol_factor_cluster(int64_t n, int W, int C, const int64_t* __restrict__ Ap,
                       const int64_t* __restrict__ Ar, const double* __restrict__ Av,
                       const double* __restrict__ d0, const double* __restrict__ rsum,
                       int* level, int64_t* Lp, int64_t* Lr, double* Lv, int64_t cap,
                       double discard, int64_t max_nnz, double rel_discard, int diag_keep,
                       int64_t* result) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char cl_smem[];
    __shared__ int64_t s_nnz;
    __shared__ int s_cn, s_nown, s_np, s_levj, s_kept, s_owner, s_fail;
    __shared__ double s_sj;
    const ClLayout Ly = cl_layout(W, C);
    const int S = (int)Ly.S, Wp = (int)Ly.Wp;
    double* F = reinterpret_cast<double*>(cl_smem + Ly.o_F);
    double* dl = reinterpret_cast<double*>(cl_smem + Ly.o_d);
    double* kv = reinterpret_cast<double*>(cl_smem + Ly.o_kv);
    double* cL = reinterpret_cast<double*>(cl_smem + Ly.o_cL);
    int* lev = reinterpret_cast<int*>(cl_smem + Ly.o_lev);
    int* ki = reinterpret_cast<int*>(cl_smem + Ly.o_ki);
    int* ci = reinterpret_cast<int*>(cl_smem + Ly.o_ci);
    int* own = reinterpret_cast<int*>(cl_smem + Ly.o_own);
    int* pre = reinterpret_cast<int*>(cl_smem + Ly.o_pre);
    uint8_t* pat = cl_smem + Ly.o_pat;
    const int r = (int)cluster.block_rank();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    // Slot s belongs to CTA s mod C at local index s / C (interleaved, so the
    // heavy targets just below the pivot spread over the cluster). s < 449
    // and C <= 8: (s * mC) >> 16 with mC = ceil(65536 / C) is s / C exactly.
    const int mC = (65536 + C - 1) / C;
    auto divC = [mC](int v) { return (v * mC) >> 16; };

    // Initial front: columns 0 .. min(W, n) - 1 sit in slots 0 .. W - 1.
    for (int q = threadIdx.x; q < S * Wp; q += blockDim.x) {
        F[q] = 0.0;
        pat[q] = 0;
    }
    __syncthreads();
    for (int ls = warp; r + ls * C < W; ls += nw) {
        const int64_t c = r + ls * C;
        if (c >= n) continue;
        for (int64_t k = Ap[c] + lane; k < Ap[c + 1]; k += 32) {
            const int64_t i = Ar[k];
            const double v = Av[k];
            if (i > c && v != 0.0) {
                F[ls * Wp + (int)(i - c)] = v;
                pat[ls * Wp + (int)(i - c)] = 1;
            }
        }
        if (lane == 0) {
            dl[ls] = d0[c];
            lev[ls] = 0;
        }
    }
    if (threadIdx.x == 0) {
        s_nnz = 0;
        s_fail = 0;
        if (r == 0) Lp[0] = 0;
    }
    cluster.sync();

    // Last warp: A's column pointers of column j + W (loaded a column ahead)
    // and entries of column j - 1 + W (loaded at the previous column).
    int64_t pk0 = 0, pk1 = 0, ebeg = 0, eend = 0;
    int64_t ei[2] = {-1, -1};
    double ev[2] = {0.0, 0.0}, ed0 = 0.0;
    if (warp == nw - 1 && W < n) {
        pk0 = Ap[W];
        pk1 = Ap[W + 1];
    }
    double rs_next = (warp == 0) ? rsum[0] : 0.0;
    int slot = 0, pslot = W - 1;      // j % W and (j - 1) % W

    for (int64_t j = 0; j < n; ++j) {
        if (warp == 0) {
            const int lsj = divC(slot), f = slot - lsj * C;
            const double rs = rs_next;
            if (j + 1 < n) rs_next = rsum[j + 1];
            const double* Fj = cluster.map_shared_rank(F, f) + lsj * Wp;
            const uint8_t* Pj = cluster.map_shared_rank(pat, f) + lsj * Wp;
            const double dj = cluster.map_shared_rank(dl, f)[lsj];
            const int levj = cluster.map_shared_rank(lev, f)[lsj];
            // Offsets o = 1 + lane + 32 k: lane order is ascending rows, the
            // order in which the reference sorts its candidates (ichol.py:87-89).
            double a[NCH];
            bool flag[NCH];
#pragma unroll
            for (int k = 0; k < NCH; ++k) {
                const int o = 1 + lane + 32 * k;
                const bool in = o < W && j + o < n;
                a[k] = in ? Fj[o] : 0.0;
                flag[k] = in && Pj[o] != 0;
            }
            unsigned fm[NCH];
            int cn = 0;
#pragma unroll
            for (int k = 0; k < NCH; ++k) {
                fm[k] = __ballot_sync(0xffffffffu, flag[k]);
                cn += __popc(fm[k]);
            }
            const int64_t nnz = s_nnz;
            int fail = 0;
            if (!(dj > 0.0)) fail = -1;                                         // ichol.py:80-81
            else if (nnz + 1 + cn > max_nnz || nnz + 1 + cn > cap) fail = -2;   // ichol.py:82-83
            const bool owner = f == r;
            const int64_t nnz0 = nnz + 1;
            // Candidates in ascending rows: value and offset, compacted.
            int cpos = 0;
#pragma unroll
            for (int k = 0; k < NCH; ++k) {
                if (flag[k]) {
                    const int q = cpos + __popc(fm[k] & lt);
                    cL[q] = a[k];
                    ci[q] = 1 + lane + 32 * k;
                }
                cpos += __popc(fm[k]);
            }
            __syncwarp();
            int kept = 0, nown = 0;
            if (!fail) {
                const double sj = sqrt(dj);
                const double rel = rel_discard * rs;
                if (lane == 0) s_sj = sj;
                // One quotient per candidate, lane-strided (the candidates
                // of a column are a quarter of its offsets or fewer).
                for (int t0 = 0; t0 < cn; t0 += 32) {
                    const int t = t0 + lane;
                    double L = 0.0;
                    bool keep = false, mine = false;
                    int o = 0;
                    if (t < cn) {
                        const double av = cL[t];
                        o = ci[t];
                        L = av / sj;
                        keep = fabs(L) > discard && fabs(av) > rel;
                        int sl = slot + o;
                        if (sl >= W) sl -= W;
                        mine = keep && sl - divC(sl) * C == r;
                        cL[t] = L;
                        ci[t] = keep ? o : -o;
                    }
                    const unsigned km = __ballot_sync(0xffffffffu, keep);
                    const unsigned om = __ballot_sync(0xffffffffu, mine);
                    if (keep) {
                        const int pos = kept + __popc(km & lt);
                        kv[pos] = L;
                        ki[pos] = o;
                        if (mine) own[nown + __popc(om & lt)] = pos;
                    }
                    kept += __popc(km);
                    nown += __popc(om);
                }
            }
            // Exclusive prefix of the owned targets' pair counts (kept - 1 -
            // pb pairs for the target at kept index pb).
            int np = 0;
            for (int t0 = 0; t0 < nown; t0 += 32) {
                const int t = t0 + lane;
                const int cnt = t < nown ? kept - 1 - own[t] : 0;
                int incl = cnt;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += v;
                }
                if (t < nown) pre[t] = np + incl - cnt;
                np += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) {
                s_fail = fail;
                if (!fail) {
                    s_cn = cn;
                    s_nown = nown;
                    s_np = np;
                    s_levj = levj;
                    s_kept = kept;
                    s_owner = owner;
                    s_nnz = nnz0 + kept;
                }
            }
        } else if (warp == nw - 1) {
            // Recycle slot (j - 1) % W for column c = j - 1 + W (its readers
            // all passed the barrier of column j - 1).
            const int64_t c = j - 1 + W;
            const int pls = divC(pslot);
            if (j >= 1 && c < n && pslot - pls * C == r) {
                double* Fc = F + pls * Wp;
                uint8_t* Pc = pat + pls * Wp;
                for (int o = lane; o < W; o += 32) {
                    Fc[o] = 0.0;
                    Pc[o] = 0;
                }
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int64_t k = ebeg + lane + 32 * e;
                    if (k < eend && ei[e] > c && ev[e] != 0.0) {
                        Fc[ei[e] - c] = ev[e];
                        Pc[ei[e] - c] = 1;
                    }
                }
                for (int64_t k = ebeg + 64 + lane; k < eend; k += 32) {   // rows longer than 64
                    const int64_t i = Ar[k];
                    const double v = Av[k];
                    if (i > c && v != 0.0) {
                        Fc[i - c] = v;
                        Pc[i - c] = 1;
                    }
                }
                if (lane == 0) {
                    dl[pls] = ed0;
                    lev[pls] = 0;
                }
            }
            // Entries of column j + W for the next column's recycle.
            if (j + W < n) {
                ebeg = pk0;
                eend = pk1;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int64_t k = pk0 + lane + 32 * e;
                    ei[e] = k < pk1 ? Ar[k] : -1;
                    ev[e] = k < pk1 ? Av[k] : 0.0;
                }
                ed0 = d0[j + W];
            }
            // Column pointers of column j + 1 + W.
            if (j + 1 + W < n) {
                pk0 = Ap[j + 1 + W];
                pk1 = Ap[j + 2 + W];
            }
        }
        __syncthreads();
        if (s_fail) break;
        // Phase P: CTA-local updates of the rows and front columns owned here.
        // Pairs are spread evenly over the threads (target found by binary
        // search of the prefix); the diagonal and level updates go to the
        // threads with the fewest pairs.
        const int nown = s_nown, cn = s_cn, np = s_np, lj = s_levj + 1;
        // The owner of slot j writes column j of L from the kept list
        // (threads 128.., which have the fewest pairs besides the diagonal
        // and level updates).
        if (s_owner) {
            const int kept = s_kept;
            const int64_t end = s_nnz, nnz = end - kept - 1;
            for (int q = (int)((threadIdx.x + blockDim.x - 128) % blockDim.x); q <= kept;
                 q += blockDim.x) {
                if (q == 0) {
                    Lv[nnz] = s_sj;
                    Lr[nnz] = j;
                    level[j] = s_levj;
                    Lp[j + 1] = end;
                } else {
                    Lv[nnz + q] = kv[q - 1];
                    Lr[nnz + q] = j + ki[q - 1];
                }
            }
        }
        for (int p = threadIdx.x; p < np; p += blockDim.x) {
            int tl = 0, th = nown - 1;
            while (tl < th) {
                const int mid = (tl + th + 1) >> 1;
                if (pre[mid] <= p) tl = mid;
                else th = mid - 1;
            }
            const int pb = own[tl];
            const int q = pb + 1 + (p - pre[tl]);
            const int ob = ki[pb];
            int sl = slot + ob;
            if (sl >= W) sl -= W;
            const int o = ki[q] - ob;
            F[divC(sl) * Wp + o] -= kv[q] * kv[pb];
            pat[divC(sl) * Wp + o] = 1;
        }
        for (int q = (int)blockDim.x - 1 - (int)threadIdx.x; q < cn; q += blockDim.x) {
            const int code = ci[q];
            int sl = slot + (code < 0 ? -code : code);
            if (sl >= W) sl -= W;
            const int ls = divC(sl);
            if (sl - ls * C != r || (!diag_keep && code < 0)) continue;
            dl[ls] -= cL[q] * cL[q];
        }
        for (int t = (int)(threadIdx.x ^ (blockDim.x >> 1)); t < nown; t += blockDim.x) {
            int sl = slot + ki[own[t]];
            if (sl >= W) sl -= W;
            const int ls = divC(sl);
            if (lev[ls] < lj) lev[ls] = lj;
        }
        pslot = slot;
        slot = slot + 1 == W ? 0 : slot + 1;
        cluster.sync();
    }
    // No CTA leaves while another may still read its shared memory.
    cluster.sync();
    if (r == 0 && threadIdx.x == 0) *result = s_fail ? (int64_t)s_fail : s_nnz;
}

bool ichol_launch_factor_cluster(int64_t n, int64_t W, const int64_t* Ap, const int64_t* Ar,
                                 const double* Av, const double* d, const double* rsum, int* level,
                                 int64_t* Lp, int64_t* Lr, double* Lv, int64_t cap, double discard,
                                 int64_t max_nnz, double rel, int diag_keep, int64_t* result,
                                 cudaStream_t s) {
    const int C = ichol_cluster_size(W);
    if (C == 0) return false;
    const ClLayout L = cl_layout(W, C);
    const int chunks = (int)((W - 1 + 31) / 32);
    auto kern = chunks <= 8 ? k_ichol_factor_cluster<8> : k_ichol_factor_cluster<kClMaxChunks>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)C);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = L.bytes;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)C;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.bytes) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters >= 1 &&
        cudaLaunchKernelEx(&cfg, kern, n, (int)W, C, Ap, Ar, Av, d, rsum, level, Lp, Lr, Lv, cap, discard,
                           max_nnz, rel, diag_keep, result) == cudaSuccess)
        return true;
    cudaGetLastError();
    return false;
}

// The rule that the table at the head of this file gives: kept entries a column
// above which the cluster is the faster one (0: it never is).
int64_t ichol_dense_columns(int64_t W) {
    const int C = ichol_cluster_size(W);
    const int64_t m = C > 0 ? 900 / C : 0;
    return m > 0 && m < W - 1 ? m : 0;
}

}  // namespace pmb
