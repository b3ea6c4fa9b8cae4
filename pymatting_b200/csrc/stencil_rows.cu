// Row-streaming half-stencil kernels: the CG apply, the V-cycle's restriction
// and its prolongation with one post sweep, for the default cycle.
//
// A warp owns a strip of 32 V adjacent columns and walks down the rows of a
// segment. Lane j holds columns x0 + V j .. + V - 1 of everything: the five
// operand rows around the current one (with two columns on either side,
// fetched from the neighbour lanes by shuffles when the row arrives), and the
// backward entries, which are the planes of the two rows above, shifted by
// their dx once and kept. So every plane value is read from memory once per
// strip, no operand or plane is read back from shared memory at another
// lane's address, and no barrier stands between rows. The outer lanes (one on
// each side) only feed their neighbours: a strip yields 30 V columns.
//
// Rows come through a private ring: every lane copies its own V elements of
// the 13 planes and the operand rows with cp.async, kAhead rows before it
// uses them, and reads back only what it copied itself, so a wait on its own
// copy groups is the only synchronisation. This keeps about 60 KB per SM in
// flight and needs no registers for it.
//
// What bounds it: HBM (planes and vectors are read once) where an image
// fills the GPU, the instructions of a row (FP64: 431 per warp and row of the
// apply, two warps per scheduler) where one wave of units holds it all. The
// tile kernels these replaced kept a 72 x 10 box of every plane in shared
// memory and spent their time on loads of shifted entries and on the
// barriers of each tile. Level 0 of 64 images (73 Mpix, FP32), tile kernels
// and these: apply 0.70 and 0.87 of the measured copy bandwidth, restriction
// 0.56 and 0.90, prolongation 0.58 and 0.75; one V-cycle of 1920x1080 in FP64
// 352 and 310 us (251 us with the programmatic launches of pm_common.cuh).
//
// Work is cut into units of `seg` rows of one strip, kUnitWarps units per
// CTA; one CTA per entry of the unit table, so that the hardware scheduler
// balances images that are still running. Arithmetic per pixel: the order of
// the one-pixel-per-thread kernels (stencil.cu), so results are bit-identical.
#include "pm_common.cuh"
#include "stencil.cuh"

namespace pmb {

namespace {

constexpr int kAhead = 2;              // rows in flight ahead of the current one
constexpr int kRing = kAhead + 1;

constexpr int kRowCtas = 2;            // resident CTAs; the ring's shared memory allows as many
// Columns per lane: one 16-byte vector.
template <typename T> constexpr int kVec = 16 / sizeof(T);

template <typename T, int V>
__device__ __forceinline__ void copy_async(T* dst, const T* src, int n) {
    // n bytes of the V elements are read, the others are zero-filled.
    constexpr int B = sizeof(T) * V;
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    static_assert(B == 16, "cp.async.cg copies 16 bytes");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Element at column offset v + dx of a row held V per lane.
template <typename T, int V>
__device__ __forceinline__ T col_at(const T (&a)[V], int v, int dx) {
    const int i = v + dx;
    if (i >= 0 && i < V) return a[i];
    if (i < 0) {
        const int up = (-i + V - 1) / V;
        return __shfl_up_sync(0xffffffffu, a[i + up * V], up);
    }
    return __shfl_down_sync(0xffffffffu, a[i % V], i / V);
}

// Row with two columns on either side.
template <typename T, int V>
__device__ __forceinline__ void widen(const T (&a)[V], T (&e)[V + 4]) {
#pragma unroll
    for (int j = 0; j < V + 4; ++j) e[j] = col_at<T, V>(a, j - 2, 0);
}

// Where a warp's unit lies: grid, first column of the lane, rows.
struct Unit {
    int col;             // first column of this lane (may lie outside the image)
    int at;              // the same, or 0 where the lane has no column in the image
    int nv;              // columns of the lane inside the image (0 .. V)
    int cta;             // CTA's index in the unit table, and the image's range of CTAs
    int c0, c1;
    int y0, y1;          // rows of the unit
    bool active;
};

template <int V, int SW, int LEAD>
__device__ __forceinline__ Unit unit_of(const RowList& R, const int4& d, int cta, const GridDesc& g,
                                        int rows) {
    Unit u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = d.y + warp;
    u.active = k < d.w;
    const int seg = k / d.z, strip = k - seg * d.z;
    const int x0 = strip * SW - LEAD * V;
    u.col = x0 + lane * V;
    u.nv = u.col < 0 ? 0 : max(0, min(V, g.w - u.col));
    u.at = u.nv > 0 ? u.col : 0;
    u.cta = cta;
    u.c0 = cta - d.y / kUnitWarps;
    u.c1 = u.c0 + (d.w + kUnitWarps - 1) / kUnitWarps;
    u.y0 = seg * R.seg;
    u.y1 = min(u.y0 + R.seg, rows);
    return u;
}

// V elements of row y of a pitched array (zero outside the image). MUT: the
// array is written by other kernels of the chain.
template <typename T, int V, bool MUT>
__device__ __forceinline__ void load_row(const T* base, int pitch, int y, int h, const Unit& u,
                                         T (&o)[V]) {
#pragma unroll
    for (int v = 0; v < V; ++v) o[v] = T(0);
    if (u.nv > 0 && y >= 0 && y < h) {
        if (MUT) ldv_l2<T, V>(base + (int64_t)y * pitch + u.col, o);
        else ldv<T, V>(base + (int64_t)y * pitch + u.col, o);
#pragma unroll
        for (int v = 1; v < V; ++v)
            if (v >= u.nv) o[v] = T(0);
    }
}

// Backward entries of a row: planes of the rows above, shifted by their dx.
template <typename T, int V>
struct Back {
    T b1[5][V];          // planes 3..7 of row y - 1
    T b2[5][V];          // planes 8..12 of row y - 2
    T b2n[5][V];         // planes 8..12 of row y - 1
};

template <typename T, int V>
__device__ __forceinline__ void shift_plane(const T (&c)[V], int dx, T (&o)[V]) {
#pragma unroll
    for (int v = 0; v < V; ++v) o[v] = col_at<T, V>(c, v, -dx);
}

template <typename T, int V>
__device__ __forceinline__ void back_init(Back<T, V>& B, const T* P, const GridDesc& g, int y,
                                          const Unit& u) {
    T c[V];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        load_row<T, V, false>(P + (8 + k) * g.pstride, g.pitch, y - 2, g.h, u, c);
        shift_plane<T, V>(c, k - 2, B.b2[k]);
        load_row<T, V, false>(P + (8 + k) * g.pstride, g.pitch, y - 1, g.h, u, c);
        shift_plane<T, V>(c, k - 2, B.b2n[k]);
        load_row<T, V, false>(P + (3 + k) * g.pstride, g.pitch, y - 1, g.h, u, c);
        shift_plane<T, V>(c, k - 2, B.b1[k]);
    }
}

// (A x) for the lane's V pixels of the current row, in the order of
// stencil_at (FP64) or in two chains, forward and backward (FP32). d0: plane
// 0 of the row; plane(p, o) gives planes 1..12 of the row; W: operand rows
// y - 2 .. y + 2, widened. The backward entries move on to the next row.
template <typename T, int V, typename Plane>
__device__ __forceinline__ void stencil_row(const T (&d0)[V], Plane plane, const T (&W)[5][V + 4],
                                            Back<T, V>& B, T (&acc)[V]) {
    constexpr bool kSplit = sizeof(T) == 4;
    T accb[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        acc[v] = d0[v] * W[2][2 + v];
        accb[v] = T(0);
    }
#pragma unroll
    for (int p = 1; p < kNH; ++p) {
        const int dy = half_dy(p), dx = half_dx(p);
        T f[V], b[V];
        plane(p, f);
        if (dy == 0) shift_plane<T, V>(f, dx, b);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const T bv = dy == 0 ? b[v] : (dy == 1 ? B.b1[p - 3 < 0 ? 0 : p - 3][v]
                                                   : B.b2[p - 8 < 0 ? 0 : p - 8][v]);
            acc[v] += f[v] * W[2 + dy][2 + v + dx];
            if (kSplit) accb[v] += bv * W[2 - dy][2 + v - dx];
            else acc[v] += bv * W[2 - dy][2 + v - dx];
        }
        if (dy == 1) shift_plane<T, V>(f, dx, B.b1[p - 3 < 0 ? 0 : p - 3]);
        if (dy == 2) {
#pragma unroll
            for (int v = 0; v < V; ++v) B.b2[p - 8 < 0 ? 0 : p - 8][v] = B.b2n[p - 8 < 0 ? 0 : p - 8][v];
            shift_plane<T, V>(f, dx, B.b2n[p - 8 < 0 ? 0 : p - 8]);
        }
    }
    if (kSplit) {
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] += accb[v];
    }
}

template <typename T, int N>
__device__ __forceinline__ void roll(T (&W)[5][N]) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < N; ++j) W[k][j] = W[k + 1][j];
}

// Whether an image is running, as far as can be told before grid_wait (it may
// finish, or its solve may begin, while this kernel waits); warp-uniform.
__device__ __forceinline__ bool looks_running(const InstState* s) {
    return __any_sync(0xffffffffu, *(volatile const int*)&s->status == kRunning);
}

extern __shared__ __align__(128) char r_smem[];

// The lane's slot of ring row `r`, array `k` (NA arrays of 32 V elements).
template <typename T, int V, int NA>
__device__ __forceinline__ T* ring_at(int r, int k) {
    T* base = reinterpret_cast<T*>(r_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    return base + (((warp * kRing + r) * NA + k) * 32 + lane) * V;
}

template <int V> __host__ __device__ constexpr int strip_cols() { return 30 * V; }
// Restriction: the lane left of a coarse pixel's own must hold a residual.
template <int V> __host__ __device__ constexpr int strip_coarse() { return 29 * V / 2; }

}  // namespace

// --------------------------------------------------------------------------
// p = z + beta p_old (z on the first pass), Ap = A p, p . Ap; finaliser
// alpha = rz / (p . Ap) (cg.py:85-90, 111-113). CG = false: y = A x alone.
// --------------------------------------------------------------------------

template <typename T, bool CG>
__global__ void __launch_bounds__(kUnitWarps * 32, kRowCtas)
k_rows_apply(RowList R, int rev, const T* __restrict__ Pl, const T* z, T* p0, T* p1,
             T* Ap, InstState* st, double* partials) {
    constexpr int V = kVec<T>, NA = kNH + (CG ? 2 : 1);
    __shared__ double s_red[32];
    grid_trigger();
    const int cta = rev ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
    const int4 d = R.cta[cta];
    const GridDesc g = R.grids[d.x];
    const Unit u = unit_of<V, strip_cols<V>(), 1>(R, d, cta, g, g.h);
    const T* P = Pl + g.poff;
    const int nb = u.nv * (int)sizeof(T);
    int64_t orow = (int64_t)u.y0 * g.pitch + u.at;               // next row to issue
    Back<T, V> B;
    auto planes_row = [&](int r, int64_t o) {
        T* dst = ring_at<T, V, NA>(r, 0);
#pragma unroll
        for (int p = 0; p < kNH; ++p) copy_async<T, V>(dst + p * 32 * V, P + o + p * g.pstride, nb);
    };
    auto prefetch = [&]() {
        if (!u.active) return;
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
            if (u.y0 + k < u.y1) planes_row(k, orow + k * g.pitch);
        back_init<T, V>(B, P, g, u.y0, u);
    };
    const bool early = !CG || looks_running(st + g.inst);
    if (early) prefetch();
    grid_wait();
    bool first = true;
    int par = 0;
    T beta = T(0);
    if (CG) {
        const volatile InstState* s = st + g.inst;
        if (s->status != kRunning) {
            copy_wait_all();
            return;
        }
        first = (s->flags & kFirst) != 0;
        par = s->iters & 1;
        beta = (T)s->beta;
    }
    if (!early) prefetch();
    double sum[1] = {0.0};
    if (u.active) {
        const T* Z = z + g.voff;
        const T* Q = (par ? p1 : p0) + g.voff;
        T* pn = (par ? p0 : p1) + g.voff;
        T* ap = Ap + g.voff;
        int ri = 0;
        auto issue = [&](int y, bool pl) {
            if (y < u.y1) {
                if (pl) planes_row(ri, orow);
                T* dst = ring_at<T, V, NA>(ri, 0);
                const bool ok = y + 2 < g.h;
                const int64_t o2 = ok ? orow + 2 * g.pitch : orow;
                copy_async<T, V>(dst + kNH * 32 * V, Z + o2, ok ? nb : 0);
                if (CG && !first) copy_async<T, V>(dst + (kNH + 1) * 32 * V, Q + o2, ok ? nb : 0);
                orow += g.pitch;
                ri = ri + 1 == kRing ? 0 : ri + 1;
            }
            copy_commit();
        };
#pragma unroll
        for (int k = 0; k < kAhead; ++k) issue(u.y0 + k, false);
        T W[5][V + 4];
        auto operand = [&](T (&zv)[V], const T (&qv)[V]) {
            if (CG && !first) {
#pragma unroll
                for (int v = 0; v < V; ++v) zv[v] = zv[v] + beta * qv[v];
            }
        };
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            T zv[V], qv[V];
            load_row<T, V, true>(Z, g.pitch, u.y0 - 2 + k, g.h, u, zv);
            if (CG && !first) load_row<T, V, true>(Q, g.pitch, u.y0 - 2 + k, g.h, u, qv);
            operand(zv, qv);
            widen<T, V>(zv, W[k + 1]);
        }
        const int lane = threadIdx.x & 31;
        const bool out = lane >= 1 && lane < 31 && u.nv > 0;
        int r = 0;
#pragma unroll 1
        for (int y = u.y0; y < u.y1; ++y) {
            issue(y + kAhead, true);
            copy_wait<kAhead>();
            roll(W);
            const T* row = ring_at<T, V, NA>(r, 0);
            T zv[V], qv[V];
            ldv<T, V>(row + kNH * 32 * V, zv);
            if (CG && !first) ldv<T, V>(row + (kNH + 1) * 32 * V, qv);
            operand(zv, qv);
            widen<T, V>(zv, W[4]);
            auto plane = [&](int p, T (&o)[V]) { ldv<T, V>(row + p * 32 * V, o); };
            T d0[V], acc[V], pv[V];
            plane(0, d0);
            stencil_row<T, V>(d0, plane, W, B, acc);
            if (out) {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    pv[v] = W[2][2 + v];
                    if (v >= u.nv) acc[v] = T(0);
                    sum[0] += (double)pv[v] * (double)acc[v];
                }
                const int64_t i = (int64_t)y * g.pitch + u.col;
                if (CG) stv<T, V>(pn + i, pv);
                stv<T, V>(ap + i, acc);
            }
            r = r + 1 == kRing ? 0 : r + 1;
        }
        copy_wait<0>();
    }
    if (CG) {
        volatile InstState* s = st + g.inst;
        tile_reduce<1>(sum, partials, gridDim.x, u.cta, u.c0, u.c1, st + g.inst, s_red, [&](double* t) {
            s->pap = t[0];
            s->alpha = s->rz / t[0];
            s->flags = s->flags & ~kFirst;
        });
    }
}

// --------------------------------------------------------------------------
// One pre-smoothing sweep from zero, residual and full-weighting restriction
// (vcycle.py:12-36, 77-80): x1 = omega b / d, res = b - A x1,
// b_coarse = R res. Units are coarse rows and strips of 29 V / 2 coarse
// columns; the residual rows of a unit are 2 Y0 - 1 .. 2 Y1 - 1.
// --------------------------------------------------------------------------

template <typename T>
__global__ void __launch_bounds__(kUnitWarps * 32, kRowCtas)
k_rows_down(RowList R, int rev, const GridDesc* fine, const T* __restrict__ Pl,
            const T* b, T* bc, double omega, const InstState* st) {
    constexpr int V = kVec<T>, NA = kNH + 1;   // planes 1..12 of row y; plane 0 and b of row y + 2
    grid_trigger();
    const int cta = rev ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
    const int4 d = R.cta[cta];
    const GridDesc gc = R.grids[d.x];
    const GridDesc g = fine[d.x];
    const Unit u = unit_of<V, 2 * strip_coarse<V>(), 2>(R, d, cta, g, gc.h);
    const T* P = Pl + g.poff;
    const int ys = 2 * u.y0 - 1, ye = 2 * u.y1;      // residual rows ys .. ye - 1 (ye <= h)
    const int nb = u.nv * (int)sizeof(T);
    int64_t orow = (int64_t)ys * g.pitch + u.at;     // next row to issue
    T W[5][V + 4], bb[3][V], dd[4][V];
    Back<T, V> B;
    auto planes_row = [&](int r, int y, int64_t o) {
        T* dst = ring_at<T, V, NA>(r, 0);
        const bool ok = y >= 0;
        const T* prow = P + (ok ? o : (int64_t)u.at);
#pragma unroll
        for (int p = 1; p < kNH; ++p)
            copy_async<T, V>(dst + p * 32 * V, prow + p * g.pstride, ok ? nb : 0);
        const bool ok2 = y + 2 < g.h;
        copy_async<T, V>(dst, P + (ok2 ? o + 2 * g.pitch : (int64_t)u.at), ok2 ? nb : 0);
    };
    // Planes of the first rows: before the wait for the kernel that writes b.
    auto prefetch = [&]() {
        if (!u.active) return;
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
            if (ys + k < ye) planes_row(k, ys + k, orow + k * g.pitch);
#pragma unroll
        for (int k = 0; k < 4; ++k) load_row<T, V, false>(P, g.pitch, ys - 2 + k, g.h, u, dd[k]);
        back_init<T, V>(B, P, g, ys, u);
    };
    const bool early = !st || looks_running(st + g.inst);
    if (early) prefetch();
    grid_wait();
    if (st && __ldcg(&st[g.inst].status) != kRunning) {
        copy_wait_all();
        return;
    }
    if (!u.active) return;
    if (!early) prefetch();
    const T* bf = b + g.voff;
    int ri = 0;
    auto issue = [&](int y, bool pl) {
        if (y < ye) {
            if (pl) planes_row(ri, y, orow);
            const bool ok2 = y + 2 < g.h;
            copy_async<T, V>(ring_at<T, V, NA>(ri, kNH), bf + (ok2 ? orow + 2 * g.pitch : (int64_t)u.at),
                             ok2 ? nb : 0);
            orow += g.pitch;
            ri = ri + 1 == kRing ? 0 : ri + 1;
        }
        copy_commit();
    };
#pragma unroll
    for (int k = 0; k < kAhead; ++k) issue(ys + k, false);
    auto sweep = [&](const T (&bv)[V], const T (&dv)[V], int y, T (&x1)[V]) {
#pragma unroll
        for (int v = 0; v < V; ++v)
            x1[v] = (y >= 0 && y < g.h && v < u.nv)
                        ? smooth_div<T>((T)omega * bv[v], dv[v]) : T(0);
    };
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        T bv[V], x1[V];
        load_row<T, V, true>(bf, g.pitch, ys - 2 + k, g.h, u, bv);
        sweep(bv, dd[k], ys - 2 + k, x1);
        widen<T, V>(x1, W[k + 1]);
        if (k >= 2) {
#pragma unroll
            for (int v = 0; v < V; ++v) bb[k - 1][v] = bv[v];
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
        dd[1][v] = dd[2][v];                         // dd[k] is the row bb[k] is
        dd[2][v] = dd[3][v];
    }
    const int lane = threadIdx.x & 31;
    const int X = u.col >> 1;
    const bool out = lane >= 2 && lane < 31 && X < gc.w;
    T r0[V + 1], r1[V + 1], r2[V + 1];               // residual rows y, y - 1, y - 2
#pragma unroll
    for (int j = 0; j <= V; ++j) r0[j] = r1[j] = T(0);
    int r = 0;
#pragma unroll 1
    for (int y = ys; y < ye; ++y) {
        issue(y + kAhead, true);
        copy_wait<kAhead>();
        roll(W);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            bb[0][v] = bb[1][v];
            bb[1][v] = bb[2][v];
            dd[0][v] = dd[1][v];
            dd[1][v] = dd[2][v];
        }
        const T* row = ring_at<T, V, NA>(r, 0);
        T x1[V];
        ldv<T, V>(row + kNH * 32 * V, bb[2]);
        ldv<T, V>(row, dd[2]);
        sweep(bb[2], dd[2], y + 2, x1);
        widen<T, V>(x1, W[4]);
        auto plane = [&](int p, T (&o)[V]) { ldv<T, V>(row + p * 32 * V, o); };
        T acc[V], res[V];
        stencil_row<T, V>(dd[0], plane, W, B, acc);
#pragma unroll
        for (int v = 0; v < V; ++v)
            res[v] = (y >= 0 && v < u.nv) ? bb[0][v] - acc[v] : T(0);
#pragma unroll
        for (int j = 0; j <= V; ++j) {
            r2[j] = r1[j];
            r1[j] = r0[j];
        }
#pragma unroll
        for (int j = 0; j <= V; ++j) r0[j] = col_at<T, V>(res, j - 1, 0);
        if ((y & 1) && y > ys && out) {
            const int Y = (y - 1) >> 1;
            T o[V / 2];
#pragma unroll
            for (int k = 0; k < V / 2; ++k) {
                T s = T(0);
#pragma unroll
                for (int ax = 0; ax < 3; ++ax) s += (T)((ax == 1 ? 2.0 : 1.0) / 16.0) * r2[2 * k + ax];
#pragma unroll
                for (int ax = 0; ax < 3; ++ax) s += (T)((ax == 1 ? 4.0 : 2.0) / 16.0) * r1[2 * k + ax];
#pragma unroll
                for (int ax = 0; ax < 3; ++ax) s += (T)((ax == 1 ? 2.0 : 1.0) / 16.0) * r0[2 * k + ax];
                o[k] = s;
            }
            T* dst = bc + gc.voff + (int64_t)Y * gc.pitch + X;
#pragma unroll
            for (int k = 0; k < V / 2; ++k)
                if (X + k < gc.w) dst[k] = o[k];
        }
        r = r + 1 == kRing ? 0 : r + 1;
    }
    copy_wait<0>();
}

// --------------------------------------------------------------------------
// Prolongation and one post-smoothing sweep (vcycle.py:95-98): x2 = x1 + P xc
// with x1 = omega b / d, x3 = x2 + omega (b - A x2) / d; at level 0 also
// r . z with r = b (and (r - r_old) . z) and beta.
// --------------------------------------------------------------------------

template <typename T>
__global__ void __launch_bounds__(kUnitWarps * 32, kRowCtas)
k_rows_up(RowList R, int rev, const GridDesc* coarse, const T* __restrict__ Pl,
          const T* b, const T* xc, T* xout, double omega, InstState* st,
          int level0, const T* dr, int reorth, double* partials) {
    // Ring row y: planes 1..12 of row y; plane 0 and b of row y + 2. The
    // second parent row of row y + 2 comes through registers, one row ahead.
    // A lane needs coarse columns X .. X + V / 2.
    constexpr int V = kVec<T>, NA = kNH + 1, NC = V / 2 + 1;
    __shared__ double s_red[2 * 32];
    grid_trigger();
    const int cta = rev ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
    const int4 d = R.cta[cta];
    const GridDesc g = R.grids[d.x];
    const GridDesc gc = coarse[d.x];
    const Unit u = unit_of<V, strip_cols<V>(), 1>(R, d, cta, g, g.h);
    const T* P = Pl + g.poff;
    const int nb = u.nv * (int)sizeof(T);
    int64_t orow = (int64_t)u.y0 * g.pitch + u.at;               // next row to issue
    T W[5][V + 4], bb[3][V], dd[4][V];
    Back<T, V> B;
    auto planes_row = [&](int r, int y, int64_t o) {
        T* dst = ring_at<T, V, NA>(r, 0);
#pragma unroll
        for (int p = 1; p < kNH; ++p) copy_async<T, V>(dst + p * 32 * V, P + o + p * g.pstride, nb);
        const bool ok2 = y + 2 < g.h;
        copy_async<T, V>(dst, P + (ok2 ? o + 2 * g.pitch : o), ok2 ? nb : 0);
    };
    // Planes of the first rows: before the wait for the kernel that writes xc.
    auto prefetch = [&]() {
        if (!u.active) return;
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
            if (u.y0 + k < u.y1) planes_row(k, u.y0 + k, orow + k * g.pitch);
#pragma unroll
        for (int k = 0; k < 4; ++k) load_row<T, V, false>(P, g.pitch, u.y0 - 2 + k, g.h, u, dd[k]);
        back_init<T, V>(B, P, g, u.y0, u);
    };
    const bool early = !st || looks_running(st + g.inst);
    if (early) prefetch();
    grid_wait();
    if (st && __ldcg(&st[g.inst].status) != kRunning) {
        copy_wait_all();
        return;
    }
    if (!early) prefetch();
    double sum[2] = {0.0, 0.0};
    if (u.active) {
        const T* bf = b + g.voff;
        const T* cf = xc + gc.voff;
        T* xo = xout + g.voff;
        const int X = u.col >> 1;
        bool cok[NC];
#pragma unroll
        for (int j = 0; j < NC; ++j) cok[j] = X + j >= 0 && X + j < gc.w;
        int ri = 0;
        auto issue = [&](int y, bool pl) {
            if (y < u.y1) {
                if (pl) planes_row(ri, y, orow);
                const bool ok2 = y + 2 < g.h;
                copy_async<T, V>(ring_at<T, V, NA>(ri, kNH), bf + (ok2 ? orow + 2 * g.pitch : orow),
                                 ok2 ? nb : 0);
                orow += g.pitch;
                ri = ri + 1 == kRing ? 0 : ri + 1;
            }
            copy_commit();
        };
#pragma unroll
        for (int k = 0; k < kAhead; ++k) issue(u.y0 + k, false);
        T ca[NC], cb[NC], cnext[NC];                 // parent rows of the newest row, and next
        auto coarse_row = [&](int Y, T (&c)[NC]) {
#pragma unroll
            for (int j = 0; j < NC; ++j)
                c[j] = cok[j] && Y >= 0 && Y < gc.h ? __ldcg(cf + (int64_t)Y * gc.pitch + X + j) : T(0);
        };
        // x2 of row y from b, plane 0 and its parent rows: an even coordinate
        // has one parent (weight 2), an odd one two (weight 1); the second
        // parent of an even row enters with weight 0.
        auto prolong = [&](const T (&bv)[V], const T (&dv)[V], int y, T (&x2)[V]) {
            const int oy = y & 1;
            const T wy0 = T(2 - oy), wy1 = T(oy), s16 = T(0.0625);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                T val = T(0);
                if (y >= 0 && y < g.h && v < u.nv) {
                    const T x1 = smooth_div<T>((T)omega * bv[v], dv[v]);
                    const int j = v >> 1;
                    const T wx0 = T(2 - (v & 1));
                    T s = T(0);
                    s += (wx0 * wy0 * s16) * ca[j];
                    if (v & 1) s += (wy0 * s16) * ca[j + 1];
                    s += (wx0 * wy1 * s16) * cb[j];
                    if (v & 1) s += (wy1 * s16) * cb[j + 1];
                    val = x1 + s;
                }
                x2[v] = val;
            }
        };
        coarse_row((u.y0 - 2) >> 1, cb);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int y = u.y0 - 2 + k;
            T bv[V], x2[V];
            load_row<T, V, true>(bf, g.pitch, y, g.h, u, bv);
            // Parent rows: y >> 1, and for odd rows the next one.
            T cn[NC];
            coarse_row((y + 1) >> 1, cn);
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                if (y & 1) ca[j] = cb[j];
                else ca[j] = cn[j];
                cb[j] = cn[j];
            }
            prolong(bv, dd[k], y, x2);
            widen<T, V>(x2, W[k + 1]);
            if (k >= 2) {
#pragma unroll
                for (int v = 0; v < V; ++v) bb[k - 1][v] = bv[v];
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            dd[1][v] = dd[2][v];                     // dd[k] is the row bb[k] is
            dd[2][v] = dd[3][v];
        }
        coarse_row((u.y0 + 3) >> 1, cnext);
        const int lane = threadIdx.x & 31;
        const bool out = lane >= 1 && lane < 31 && u.nv > 0;
        int r = 0;
#pragma unroll 1
        for (int y = u.y0; y < u.y1; ++y) {
            issue(y + kAhead, true);
            copy_wait<kAhead>();
            roll(W);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                bb[0][v] = bb[1][v];
                bb[1][v] = bb[2][v];
                dd[0][v] = dd[1][v];
                dd[1][v] = dd[2][v];
            }
            const T* row = ring_at<T, V, NA>(r, 0);
            ldv<T, V>(row + kNH * 32 * V, bb[2]);
            ldv<T, V>(row, dd[2]);
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                if (y & 1) ca[j] = cb[j];
                else ca[j] = cnext[j];
                cb[j] = cnext[j];
            }
            if (y + 1 < u.y1) coarse_row((y + 4) >> 1, cnext);
            T x2[V];
            prolong(bb[2], dd[2], y + 2, x2);
            widen<T, V>(x2, W[4]);
            auto plane = [&](int p, T (&o)[V]) { ldv<T, V>(row + p * 32 * V, o); };
            T ax[V], x3[V];
            stencil_row<T, V>(dd[0], plane, W, B, ax);
            if (out) {
                const int64_t i = (int64_t)y * g.pitch + u.col;
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if (v < u.nv) {
                        x3[v] = W[2][2 + v] + smooth_div<T>((T)omega * (bb[0][v] - ax[v]), dd[0][v]);
                        if (level0) {
                            sum[0] += (double)bb[0][v] * (double)x3[v];
                            if (reorth) sum[1] += (double)__ldcg(dr + g.voff + i + v) * (double)x3[v];
                        }
                    } else {
                        x3[v] = T(0);
                    }
                }
                stv<T, V>(xo + i, x3);
            }
            r = r + 1 == kRing ? 0 : r + 1;
        }
        copy_wait<0>();
    }
    if (level0 && st) {
        InstState* s = st + g.inst;
        tile_reduce<2>(sum, partials, gridDim.x, u.cta, u.c0, u.c1, s, s_red, [&](double* t) {
            if (reorth) finish_beta_reorth(s, t[0], t[1]);
            else finish_beta(s, t[0]);
        });
    }
}

// --------------------------------------------------------------------------
// Launches
// --------------------------------------------------------------------------

namespace {

template <typename T> constexpr size_t ring_bytes(int na) {
    return (size_t)kUnitWarps * kRing * na * 32 * 16;
}
template <typename T> constexpr size_t smem_apply(bool cg) { return ring_bytes<T>(kNH + (cg ? 2 : 1)); }
template <typename T> constexpr size_t smem_cycle() { return ring_bytes<T>(kNH + 1); }

template <typename K> int rows_resident(K kernel, size_t smem) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kUnitWarps * 32, smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return n < 1 ? 1 : n;
}

template <typename T> void prepare_rows_t() {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(k_rows_apply<T, true>, attr, (int)smem_apply<T>(true));
    cudaFuncSetAttribute(k_rows_apply<T, false>, attr, (int)smem_apply<T>(false));
    cudaFuncSetAttribute(k_rows_down<T>, attr, (int)smem_cycle<T>());
    cudaFuncSetAttribute(k_rows_up<T>, attr, (int)smem_cycle<T>());
}

}  // namespace

void prepare_rows() {
    prepare_rows_t<double>();
    prepare_rows_t<float>();
}

template <typename T> int rows_strip(int kind) {
    return kind == kRowsDown ? strip_coarse<kVec<T>>() : strip_cols<kVec<T>>();
}

template <typename T> int rows_resident_of(int kind) {
    return kind == kRowsApply  ? rows_resident(k_rows_apply<T, true>, smem_apply<T>(true))
           : kind == kRowsDown ? rows_resident(k_rows_down<T>, smem_cycle<T>())
                               : rows_resident(k_rows_up<T>, smem_cycle<T>());
}

template <typename T>
void launch_rows_apply(const RowList& R, int rev, const T* P, const T* z, T* p0, T* p1, T* Ap,
                       InstState* st, double* part, cudaStream_t s) {
    if (R.total <= 0) return;
    if (st)
        launch_chain(k_rows_apply<T, true>, R.total, kUnitWarps * 32, smem_apply<T>(true), s, R, rev, P,
                     z, p0, p1, Ap, st, part);
    else
        launch_chain(k_rows_apply<T, false>, R.total, kUnitWarps * 32, smem_apply<T>(false), s, R, rev,
                     P, z, p0, p1, Ap, st, part);
}

template <typename T>
void launch_rows_down(const RowList& R, int rev, const GridDesc* fine, const T* P, const T* b, T* bc,
                      double omega, const InstState* st, cudaStream_t s) {
    if (R.total <= 0) return;
    launch_chain(k_rows_down<T>, R.total, kUnitWarps * 32, smem_cycle<T>(), s, R, rev, fine, P, b, bc,
                 omega, st);
}

template <typename T>
void launch_rows_up(const RowList& R, int rev, const GridDesc* coarse, const T* P, const T* b,
                    const T* xc, T* xout, double omega, InstState* st, int level0, const T* dr,
                    int reorth, double* part, cudaStream_t s) {
    if (R.total <= 0) return;
    launch_chain(k_rows_up<T>, R.total, kUnitWarps * 32, smem_cycle<T>(), s, R, rev, coarse, P, b, xc,
                 xout, omega, st, level0, dr, reorth, part);
}

#define PMB_ROWS_INST(T)                                                                          \
    template int rows_strip<T>(int);                                                              \
    template int rows_resident_of<T>(int);                                                        \
    template void launch_rows_apply<T>(const RowList&, int, const T*, const T*, T*, T*, T*,       \
                                       InstState*, double*, cudaStream_t);                        \
    template void launch_rows_down<T>(const RowList&, int, const GridDesc*, const T*, const T*,   \
                                      T*, double, const InstState*, cudaStream_t);                \
    template void launch_rows_up<T>(const RowList&, int, const GridDesc*, const T*, const T*,     \
                                    const T*, T*, double, InstState*, int, const T*, int,         \
                                    double*, cudaStream_t);
PMB_ROWS_INST(float)
PMB_ROWS_INST(double)
#undef PMB_ROWS_INST

}  // namespace pmb
