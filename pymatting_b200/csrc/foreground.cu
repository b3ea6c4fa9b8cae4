// Multi-level foreground / background estimation (PyMatting's
// estimate_foreground_ml, pymatting/foreground/estimate_foreground_ml.py:61-183)
// on sm_100a.
//
// The reference sweeps every level with an in-place Gauss-Seidel pass in
// raster order: pixel (y, x) of iteration i reads the NEW values of (y, x-1)
// and (y-1, x) and the OLD values of (y, x+1) and (y+1, x). This file
// reproduces that order exactly, so the results are bit-identical for the same
// seed colours:
//
// * Rows are cut into strips of 32; a warp sweeps one strip for one colour
//   channel with lane j on row 32k+j, lane j handling column s-j at step s.
//   The new value of the row above comes from lane j-1's previous step by a
//   shuffle, the old value of the row below from lane j+1's current load.
//   Lane 0 reads the strip above, lane 31 the strip below, through global
//   memory.
// Levels take one of three kernels. The first levels, up to 32x32, run in one
// launch, a CTA per channel, everything in shared memory (k_fg_small). Levels
// with one or two iterations, the default above 32x32, run k_fg_pair below.
// Levels with more iterations run k_fg_sweep:
//
// * Every (iteration, strip) pair is a unit. Units are claimed from a ticket
//   counter in order, so a unit only ever waits on units that running CTAs
//   already hold. Iteration i+1 of strip k runs behind iteration i of strip
//   k+1, so all iterations of a level are in flight at once.
// * F and B live in a diagonal layout [channel][strip][step][lane], so each
//   warp's per-step loads and stores are one contiguous 512-byte row. Every
//   value is stored as {float value, uint32 epoch} in one 64-bit word. The
//   epoch is 0 for the level's starting values and i+1 for iteration i's
//   output. A reader polls until the epoch it needs appears. A 64-bit
//   relaxed store is single-copy atomic, so no fences or progress counters are
//   needed. Every wait is bounded (2 s on %globaltimer); a timeout sets an
//   error word and the kernel drains without waiting further.
// * The per-pixel terms that depend only on alpha (the four neighbour weights
//   and the inverse of the 2x2 system) are computed once per level by a
//   parallel prep kernel. They are stored per (strip, 32-step chunk) as one
//   contiguous record that the sweep brings into shared memory with bulk
//   async copies, two chunks in flight. The F/B rows a step reads are copied
//   into a per-warp shared-memory ring kDist steps ahead (cp.async groups),
//   so each step waits only for its own rows.
//
// Arithmetic follows numba's typing of the reference (a00, da and the
// right-hand side in float32; a1, a01, a11, the determinant and the inverse
// in float64) with explicitly rounded intrinsics, so nothing is contracted
// into fused multiply-adds.

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "tma.cuh"

namespace pmb {
namespace fg {

constexpr int kLanes = 32;
constexpr int kChunk = 32;  // diagonal steps per staged coefficient chunk
constexpr int kMaxDepth = 8;
constexpr int kMaxLevels = 40;
constexpr int kGroupMax = 4;   // colour channels (warps) per sweep CTA
constexpr int kRingSlots = 8;  // shared-memory slots of F/B rows per warp
constexpr int kDist = 2;       // steps between a row's copy and its use (measured best)
constexpr unsigned long long kTimeoutNs = 2000000000ull;
constexpr int kMeanBlocks = 1184;
constexpr int kMeanThreads = 256;
constexpr int kMaxSide = 65535;
enum : int { kErrTimeout = 1, kErrStage = 2 };

// Coefficient record of one (strip, chunk): 32 steps x 32 lanes of
//   float4 da             (weights of the left, right, upper, lower neighbour)
//   double2 {b00, b01}, double b11  (inverse of the 2x2 system)
//   float2 pI[depth]      (a0 * I_c, float32(a1 * I_c))
constexpr int kOffDa = 0;
constexpr int kOffB0 = kChunk * kLanes * 16;
constexpr int kOffB11 = kOffB0 + kChunk * kLanes * 16;
constexpr int kOffPI = kOffB11 + kChunk * kLanes * 8;
constexpr int kPIBytes = kChunk * kLanes * 8;
constexpr int kBaseBytes = kOffPI;  // da and the 2x2 inverse, shared by all channels
__host__ __device__ constexpr int rec_bytes(int depth) { return kOffPI + depth * kPIBytes; }
// Shared memory of one staged chunk for a CTA of `cpg` channels.
__host__ __device__ constexpr int stage_bytes(int cpg) { return kBaseBytes + cpg * kPIBytes; }
// Per-warp ring: kRingSlots x (32 right-hand values + 32 neighbour-strip
// values, of which lanes 0 and 31 use theirs).
constexpr int kRingRow = 2 * kLanes;
constexpr int kWarpRingBytes = kRingSlots * kRingRow * 16;

struct Level {
    int h, w;    // level size
    int S, Q;    // strips, 32-step chunks per strip
    int Sp;      // steps per strip row in the diagonal layout (32 Q >= w + 31)
    int n_iter;  // Gauss-Seidel sweeps on this level
    int tagged;  // F/B kept as {value, epoch} pairs (k_fg_sweep), else as float2
};

__device__ __forceinline__ uint64_t pack(float v, uint32_t epoch) {
    return ((uint64_t)epoch << 32) | (uint64_t)__float_as_uint(v);
}
__device__ __forceinline__ float value_of(uint64_t u) { return __uint_as_float((uint32_t)u); }
__device__ __forceinline__ uint32_t epoch_of(uint64_t u) { return (uint32_t)(u >> 32); }

__device__ __forceinline__ ulonglong2 ld_fb(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ void st_fb(ulonglong2* p, uint64_t a, uint64_t b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b)
                 : "memory");
}
__device__ __forceinline__ int ld_err(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Poll until both words of *p carry `want` and return them. Bounded: gives
// up (returning the last read) when the error word is set or after
// kTimeoutNs, which it reports.
__device__ __noinline__ ulonglong2 poll_epoch(const ulonglong2* p, uint32_t want, int* err,
                                              unsigned long long timeout_ns = kTimeoutNs) {
    unsigned long long t0 = 0;
    ulonglong2 v = make_ulonglong2(0, 0);
    for (uint32_t n = 0;; ++n) {
        if ((n & 63) == 0) {
            if (ld_err(err)) return v;
            if (n == 0) {
                t0 = now_ns();
            } else if (now_ns() - t0 > timeout_ns) {
                atomicCAS(err, 0, kErrTimeout);
                return v;
            }
        }
        v = ld_fb(p);
        if (epoch_of(v.x) == want && epoch_of(v.y) == want) return v;
    }
}

__device__ __forceinline__ bool has_epoch(ulonglong2 v, uint32_t want) {
    return epoch_of(v.x) == want && epoch_of(v.y) == want;
}

// 16-byte global -> shared copy cached in L2 only, tracked by commit groups.
// With n = 0 nothing is read and the 16 bytes are zero-filled.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t n) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Named barrier 1 over the CTA's `nthreads` threads.
__device__ __forceinline__ void bar_sync1(int nthreads) {
    asm volatile("barrier.sync 1, %0;" ::"r"(nthreads) : "memory");
}

// ---------------------------------------------------------------------------
// Seed colours: mean image colour over alpha > 0.9 (foreground) and
// alpha < 0.1 (background), estimate_foreground_ml.py:79-95. Sums are taken
// in float64 in a fixed order (deterministic); the reference accumulates a
// running float32 sum, so the seeds agree to float32 rounding, not bitwise.
// ---------------------------------------------------------------------------

constexpr int kMeanValues = 2 * kMaxDepth + 2;  // F sums, B sums, F count, B count

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(kMeanThreads) k_fg_mean_partial(const float* __restrict__ image,
                                                                  const float* __restrict__ alpha,
                                                                  long long n, int depth,
                                                                  double* __restrict__ part) {
    double acc[kMeanValues];
#pragma unroll
    for (int v = 0; v < kMeanValues; ++v) acc[v] = 0.0;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
         p += (long long)gridDim.x * blockDim.x) {
        const float a = alpha[p];
        if (a > 0.9f) {
#pragma unroll
            for (int c = 0; c < kMaxDepth; ++c)
                if (c < depth) acc[c] += (double)image[p * depth + c];
            acc[2 * kMaxDepth] += 1.0;
        } else if (a < 0.1f) {
#pragma unroll
            for (int c = 0; c < kMaxDepth; ++c)
                if (c < depth) acc[kMaxDepth + c] += (double)image[p * depth + c];
            acc[2 * kMaxDepth + 1] += 1.0;
        }
    }
    __shared__ double red[kMeanThreads / 32][kMeanValues];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int v = 0; v < kMeanValues; ++v) {
        const double t = warp_sum(acc[v]);
        if (lane == 0) red[warp][v] = t;
    }
    __syncthreads();
    if (threadIdx.x < kMeanValues) {
        double t = 0.0;
        for (int wv = 0; wv < kMeanThreads / 32; ++wv) t += red[wv][threadIdx.x];
        part[(long long)blockIdx.x * kMeanValues + threadIdx.x] = t;
    }
}

// One warp per summed value, fixed order: deterministic.
__global__ void __launch_bounds__(32 * kMeanValues) k_fg_mean_final(const double* __restrict__ part,
                                                                    int nblocks, int depth,
                                                                    float* __restrict__ seed) {
    __shared__ double tot[kMeanValues];
    const int v = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double a = 0.0;
    for (int b = lane; b < nblocks; b += 32) a += part[(long long)b * kMeanValues + v];
    a = warp_sum(a);
    if (lane == 0) tot[v] = a;
    __syncthreads();
    if (threadIdx.x < depth) {
        const int c = threadIdx.x;
        seed[c] = (float)(tot[c] / (tot[2 * kMaxDepth] + 1e-5));
        seed[depth + c] = (float)(tot[kMaxDepth + c] / (tot[2 * kMaxDepth + 1] + 1e-5));
    }
}

// ---------------------------------------------------------------------------
// Prep: coefficients of one level and its starting F/B (epoch 0), both in
// the diagonal layout. The level's image and alpha are the nearest-neighbour
// resize of the input (estimate_foreground_ml.py:5-55, x_src = x w_src / w),
// the starting F/B the nearest-neighbour resize of the previous level's
// result (or the seed colours for the 1x1 level).
// ---------------------------------------------------------------------------

struct PrepArgs {
    const float* image;  // (h0, w0, depth)
    const float* alpha;  // (h0, w0)
    int h0, w0, depth;
    float reg, gw;
    Level L, P;                 // this level and the previous one (P.h == 0: seed)
    const void* fb_prev;        // previous level, diagonal layout
    const float* seed;          // F[depth], B[depth]
    unsigned char* rec;
    void* fb;                   // starting values (epoch 0 where tagged)
    uint64_t* mid;              // not tagged: the first iteration's results, unset
    uint64_t* bnd;              // not tagged: the strips' last rows, unset
    float2* dn;                 // not tagged: the row below each strip, by the step that reads it
};

// Coefficients of pixel (y, x) of level L: neighbour weights, the inverse
// {b00, b01}, b11 of its 2x2 system, and where its colours lie in the input.
struct Coef {
    float4 da;
    double b00, b01, b11;
    float a0;
    double a1;
    long long pc;
};

// x_src = x * n_src / n_dst (sides <= 65535, so the product fits 32 bits).
__device__ __forceinline__ int src_index(int v, int n_dst, int n_src) {
    if (n_dst == n_src) return v;
    const unsigned s = (unsigned)v * (unsigned)n_src / (unsigned)n_dst;
    return (int)min(s, (unsigned)(n_src - 1));
}

__device__ __forceinline__ Coef coef_at(const float* __restrict__ alpha, int h0, int w0, float reg,
                                        float gw, const Level& L, int y, int x) {
    Coef c;
    const int yc = src_index(y, L.h, h0), xc = src_index(x, L.w, w0);
    const int ym = src_index(max(y - 1, 0), L.h, h0);
    const int yp = src_index(min(y + 1, L.h - 1), L.h, h0);
    const int xm = src_index(max(x - 1, 0), L.w, w0);
    const int xp = src_index(min(x + 1, L.w - 1), L.w, w0);
    c.pc = (long long)yc * w0 + xc;
    c.a0 = alpha[c.pc];
    const float an[4] = {alpha[(long long)yc * w0 + xm], alpha[(long long)yc * w0 + xp],
                         alpha[(long long)ym * w0 + xc], alpha[(long long)yp * w0 + xc]};
    c.a1 = __dsub_rn(1.0, (double)c.a0);
    float a00 = __fmul_rn(c.a0, c.a0);
    const double a01 = __dmul_rn((double)c.a0, c.a1);
    double a11 = __dmul_rn(c.a1, c.a1);
    float d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float g = fabsf(__fsub_rn(c.a0, an[q]));
        d[q] = __fadd_rn(reg, __fmul_rn(gw, g));
        a00 = __fadd_rn(a00, d[q]);
        a11 = __dadd_rn(a11, (double)d[q]);
    }
    const double det = __dsub_rn(__dmul_rn((double)a00, a11), __dmul_rn(a01, a01));
    const double inv = __ddiv_rn(1.0, det);
    c.b00 = __dmul_rn(inv, a11);
    c.b01 = __dmul_rn(inv, -a01);
    c.b11 = __dmul_rn(inv, (double)a00);
    c.da = make_float4(d[0], d[1], d[2], d[3]);
    return c;
}
// The data term of a channel: (a0 I, float32(a1 I)).
__device__ __forceinline__ float2 data_term(const Coef& c, float I) {
    return make_float2(__fmul_rn(c.a0, I), __double2float_rn(__dmul_rn(c.a1, (double)I)));
}

// Coefficients of a level that is not tagged: planes over the diagonal
// entries (k, s, j) of the level.
struct Planes {
    float4* da;
    double2* b0;
    double* b11;
    float2* pi;        // depth planes
    long long n;       // entries
};
__host__ __device__ inline Planes planes_of(unsigned char* rec, const Level& L) {
    Planes p;
    p.n = (long long)L.S * L.Sp * kLanes;
    p.da = reinterpret_cast<float4*>(rec);
    p.b0 = reinterpret_cast<double2*>(rec + 16 * p.n);
    p.b11 = reinterpret_cast<double*>(rec + 32 * p.n);
    p.pi = reinterpret_cast<float2*>(rec + 40 * p.n);
    return p;
}

constexpr uint64_t kUnset = ~0ull;     // no F, B pair: values are clamped to [0, 1]

__device__ __forceinline__ uint64_t pack_fb(float f, float b) {
    return ((uint64_t)__float_as_uint(b) << 32) | (uint64_t)__float_as_uint(f);
}
__device__ __forceinline__ float2 unpack_fb(uint64_t u) {
    return make_float2(__uint_as_float((uint32_t)u), __uint_as_float((uint32_t)(u >> 32)));
}

// grid: (ceil(Sp * 32 / 256), S); one thread per diagonal entry (k, s, j).
__global__ void __launch_bounds__(256) k_fg_prep(PrepArgs A) {
    const Level L = A.L;
    const long long plane = (long long)L.S * L.Sp * kLanes;
    const int e_strip = blockIdx.x * blockDim.x + threadIdx.x;
    if (e_strip >= L.Sp * kLanes) return;
    const int j = e_strip & 31;
    const int s = e_strip >> 5;
    const int k = blockIdx.y;
    const long long idx = (long long)k * L.Sp * kLanes + e_strip;
    const int y = kLanes * k + j, x = s - j;
    const bool valid = y < L.h && x >= 0 && x < L.w;
    Coef co;
    co.da = make_float4(0.f, 0.f, 0.f, 0.f);
    co.b00 = co.b01 = co.b11 = 0.0;
    if (valid) co = coef_at(A.alpha, A.h0, A.w0, A.reg, A.gw, L, y, x);
    // starting values
    long long src = -1;
    if (valid && A.P.h > 0) {
        const int yq = src_index(y, L.h, A.P.h), xq = src_index(x, L.w, A.P.w);
        src = ((long long)(yq >> 5) * A.P.Sp + (xq + (yq & 31))) * kLanes + (yq & 31);
    }
    const long long pplane = (long long)A.P.S * A.P.Sp * kLanes;
    unsigned char* R = A.rec + ((long long)k * L.Q + (s >> 5)) * rec_bytes(A.depth);
    const int e = ((s & 31) << 5) | j;      // entry within the record (tagged)
    const Planes pl = planes_of(A.rec, L);
    if (L.tagged) {
        *(float4*)(R + kOffDa + e * 16) = co.da;
        *(double2*)(R + kOffB0 + e * 16) = make_double2(co.b00, co.b01);
        *(double*)(R + kOffB11 + e * 8) = co.b11;
    } else {
        pl.da[idx] = co.da;
        pl.b0[idx] = make_double2(co.b00, co.b01);
        pl.b11[idx] = co.b11;
    }
    for (int c = 0; c < A.depth; ++c) {
        float2 pi = make_float2(0.f, 0.f), v = make_float2(0.f, 0.f);
        if (valid) {
            pi = data_term(co, A.image[co.pc * A.depth + c]);
            if (src < 0) {
                v = make_float2(A.seed[c], A.seed[A.depth + c]);
            } else if (A.P.tagged) {
                const ulonglong2 u = static_cast<const ulonglong2*>(A.fb_prev)[c * pplane + src];
                v = make_float2(value_of(u.x), value_of(u.y));
            } else {
                v = static_cast<const float2*>(A.fb_prev)[c * pplane + src];
            }
        }
        if (L.tagged) {
            *(float2*)(R + kOffPI + c * kPIBytes + e * 8) = pi;
            static_cast<ulonglong2*>(A.fb)[c * plane + idx] = make_ulonglong2(pack(v.x, 0u), pack(v.y, 0u));
        } else {
            pl.pi[c * plane + idx] = pi;
            static_cast<float2*>(A.fb)[c * plane + idx] = v;
            if (L.n_iter == 2) A.mid[c * plane + idx] = kUnset;
            if (j == 0 && k > 0 && x < L.w) A.dn[((long long)c * L.S + k - 1) * L.Sp + x + 31] = v;
        }
    }
    if (!L.tagged && j == 31 && x >= 0 && x < L.w)
        for (int q = 0; q < 2 * A.depth; ++q) A.bnd[((long long)q * L.S + k) * L.Sp + x] = kUnset;
}

// ---------------------------------------------------------------------------
// Small levels: the first levels up to 32 x 32, one CTA per colour channel
// (channels do not meet), all levels in one launch. A warp per iteration
// runs the wavefront over the level's diagonal rows in shared memory, two
// steps behind the iteration before it. What bounds it is the chain of steps
// (w + 31 + 2 n_iter a level, about 0.2 us each): 97 us for the six levels of
// a 1920x1080 call, 215 us as two launches per level with every iteration in a
// CTA of its own.
// ---------------------------------------------------------------------------

constexpr int kSmallSide = 32, kSmallIters = 16, kSmallLevels = 8;
constexpr int kSmallRows = kSmallSide + kLanes;       // rows 0 .. w + 31

struct SmallArgs {
    const float* image;
    const float* alpha;
    int h0, w0, depth;
    float reg, gw;
    int n;                       // levels
    Level lv[kSmallLevels];
    const float* seed;
    float2* out;                 // last of them, diagonal layout
    int* err;
};

struct SmallSmem {
    float4 da[kSmallRows * kLanes];
    double2 b0[kSmallRows * kLanes];
    double b11[kSmallRows * kLanes];
    float2 pi[kSmallRows * kLanes];
    float2 v[(kSmallRows + 1) * kLanes];
    float2 prev[kSmallSide * kSmallSide];
    volatile int done[kSmallIters];
};

// One pixel: the reference's sums in order (left, right, upper, lower), the
// 2x2 solve and the clamp. The clamp follows the rounding to float32: that
// rounding is monotone and keeps 0 and 1, so the result is the same; NaN
// becomes 1 and -0 becomes 0, as max(0.0, min(1.0, v)) makes them.
__device__ __forceinline__ float2 fg_pixel(float2 pI, float4 da, double2 b0, double b11, float2 l,
                                           float2 r, float2 u, float2 d) {
    float f0 = pI.x, f1 = pI.y;
    f0 = __fadd_rn(f0, __fmul_rn(da.x, l.x));
    f1 = __fadd_rn(f1, __fmul_rn(da.x, l.y));
    f0 = __fadd_rn(f0, __fmul_rn(da.y, r.x));
    f1 = __fadd_rn(f1, __fmul_rn(da.y, r.y));
    f0 = __fadd_rn(f0, __fmul_rn(da.z, u.x));
    f1 = __fadd_rn(f1, __fmul_rn(da.z, u.y));
    f0 = __fadd_rn(f0, __fmul_rn(da.w, d.x));
    f1 = __fadd_rn(f1, __fmul_rn(da.w, d.y));
    const double Fc = __dadd_rn(__dmul_rn(b0.x, (double)f0), __dmul_rn(b0.y, (double)f1));
    const double Bc = __dadd_rn(__dmul_rn(b0.y, (double)f0), __dmul_rn(b11, (double)f1));
    return make_float2(fmaxf(fminf(__double2float_rn(Fc), 1.f), 0.f),
                       fmaxf(fminf(__double2float_rn(Bc), 1.f), 0.f));
}

__device__ __forceinline__ float2 shfl_up2(float2 a) {
    return make_float2(__shfl_up_sync(0xffffffffu, a.x, 1), __shfl_up_sync(0xffffffffu, a.y, 1));
}
__device__ __forceinline__ float2 shfl_down2(float2 a) {
    return make_float2(__shfl_down_sync(0xffffffffu, a.x, 1), __shfl_down_sync(0xffffffffu, a.y, 1));
}

__device__ __forceinline__ int ld_cnt(const volatile int* p) {
    const int v = *p;
    asm volatile("" ::: "memory");
    return v;
}

// Wait until the counter in shared memory reaches `want` (every lane reads
// the same word). Bounded by time and by the error word; false: give up.
__device__ __forceinline__ bool wait_cnt(const volatile int* p, int want, int* err) {
    unsigned long long t0 = 0;
    for (uint32_t n = 1;; ++n) {
        if (ld_cnt(p) >= want) return true;
        if ((n & 255) == 0) {
            if (ld_err(err)) return false;
            if (n == 256) {
                t0 = now_ns();
            } else if (now_ns() - t0 > kTimeoutNs) {
                atomicCAS(err, 0, kErrTimeout);
                return false;
            }
        }
    }
}

// Publish a counter after this warp's earlier shared-memory accesses.
__device__ __forceinline__ void put_cnt(volatile int* p, int v) {
    __threadfence_block();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) *p = v;
}

__global__ void __launch_bounds__(kLanes * kSmallIters, 1) k_fg_small(SmallArgs A) {
    extern __shared__ __align__(128) unsigned char smem[];
    SmallSmem& M = *reinterpret_cast<SmallSmem*>(smem);
    const int c = blockIdx.x, tid = threadIdx.x, nthr = blockDim.x;
    const int warp = tid >> 5, j = tid & 31;
    for (int l = 0; l < A.n; ++l) {
        const Level L = A.lv[l];
        const int T = L.w + kLanes - 1;                    // steps
        for (int q = tid; q < kSmallRows * kLanes; q += nthr) {
            const int s = q >> 5, y = q & 31, x = s - y;
            float2 v = make_float2(0.f, 0.f);
            if (y < L.h && x >= 0 && x < L.w) {
                const Coef co = coef_at(A.alpha, A.h0, A.w0, A.reg, A.gw, L, y, x);
                M.da[q] = co.da;
                M.b0[q] = make_double2(co.b00, co.b01);
                M.b11[q] = co.b11;
                M.pi[q] = data_term(co, A.image[co.pc * A.depth + c]);
                if (l == 0) v = make_float2(A.seed[c], A.seed[A.depth + c]);
                else v = M.prev[src_index(y, L.h, A.lv[l - 1].h) * kSmallSide + src_index(x, L.w, A.lv[l - 1].w)];
            }
            M.v[q] = v;
        }
        if (tid < kSmallIters) M.done[tid] = 0;
        __syncthreads();
        if (warp < L.n_iter) {
            float2 my = make_float2(0.f, 0.f), p = my;
            bool ok = true;
            for (int s = 0; s < T && ok; ++s) {
                if (warp > 0)
                    ok = __all_sync(0xffffffffu, wait_cnt(&M.done[warp - 1], min(s + 2, T), A.err));
                const int cur = s - j, q = s * kLanes + j;
                const bool in = j < L.h && cur >= 0 && cur < L.w;
                if (s == 0) p = M.v[j];
                const float2 rv = M.v[q + kLanes];
                const float2 uv = shfl_up2(my), dv = shfl_down2(rv);
                if (in) {
                    const float2 lf = cur == 0 ? p : my, rt = cur + 1 < L.w ? rv : p;
                    const float2 up = j == 0 ? p : uv, dn = j == L.h - 1 ? p : dv;
                    my = fg_pixel(M.pi[q], M.da[q], M.b0[q], M.b11[q], lf, rt, up, dn);
                    M.v[q] = my;
                }
                p = rv;
                put_cnt(&M.done[warp], s + 1);
            }
        }
        __syncthreads();
        for (int q = tid; q < T * kLanes; q += nthr) {
            const int y = q & 31, x = (q >> 5) - y;
            if (y < L.h && x >= 0 && x < L.w) {
                M.prev[y * kSmallSide + x] = M.v[q];
                if (l == A.n - 1) A.out[(long long)c * L.S * L.Sp * kLanes + q] = M.v[q];
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Levels of one or two iterations. A CTA is one colour channel and five
// warps: the first iteration on strip k, the second on strip k - 1, and three
// loaders. All that a unit waits for comes from units with smaller tickets
// (strip k - 1's first iteration, strip k - 2's second), or from inside the
// CTA: the row below strip k - 1 is strip k's first row.
//
// What bounds it is the chain of w + h diagonal steps, one pixel after
// another: a shuffle (24 cycles), three float32 operations, a float64 product
// and sum between two conversions (54), the clamp: about 105 cycles. So a
// step does little else and has no branch. Coefficients, starting values and
// the old row below come in chunks of 8 steps by bulk copies, about two chunks
// ahead; four steps' operands are in registers while the next four are
// fetched and the counters for those after are read; stores are predicated;
// and what other CTAs produce is polled by loaders, which fill rings in shared
// memory and publish counters. Results that another CTA reads carry their own
// validity: the arrays start out as kUnset, which no clamped pair can be, and
// a 64-bit relaxed store is single-copy atomic. About 245 cycles a step; with
// a CTA per (iteration, strip) that copied and polled in the step itself it was
// 640. Whole calls: 1920x1080 2.39 -> 1.63 ms, 341x227 0.69 -> 0.45 ms.
// ---------------------------------------------------------------------------

constexpr int kPairWarps = 5;
constexpr int kBlk = 4;              // steps whose operands are in registers
constexpr int kPChunk = 8;           // steps of a bulk-copied chunk
constexpr int kPSlots = 3;           // chunks in shared memory
constexpr int kInRows = 64;          // ring of the second iteration's old rows
constexpr int kAux = 64;             // ring of border values (columns)
constexpr int kRound = 16;           // rows a loader round moves

struct PairArgs {
    Level L;
    int depth;
    Planes pl;
    const float2* in;      // starting values
    const float2* dn;      // of the row below each strip, by step
    uint64_t* mid;         // first iteration's results (n_iter == 2)
    float2* out;           // last iteration's results
    uint64_t* bnd;         // last rows: [iteration][channel][strip][column]
    int* ticket;
    int* err;
};

struct PairChunk {
    float4 da[kPChunk * kLanes];
    double2 b0[kPChunk * kLanes];
    double b11[kPChunk * kLanes];
    float2 pi[kPChunk * kLanes];
};
struct PairSmem {
    PairChunk coef[2][kPSlots];
    float2 old[kPSlots][kPChunk * kLanes];       // first iteration: rows s + 1
    float2 below[kPSlots][kPChunk];              // first iteration: lane 31's lower neighbour
    float2 rows[kInRows * kLanes];               // second iteration: old rows
    float2 up[2][kAux], dn1[kAux];
    uint64_t full[2][kPSlots];
    // What a sweep waits for, read as one vector: columns of the strip above,
    // old rows or steps of the other sweep that it must not overrun, columns
    // of the row below, steps whose chunks have landed. Counters that a sweep
    // has no need of start at kNoWait.
    __align__(16) int cnt[2][4];
    volatile int done[2];
    int unit;
};
enum : int { kCntUp = 0, kCntIn = 1, kCntRing = 1, kCntDn = 2, kCntChunk = 3 };
constexpr int kNoWait = 1 << 30;

// Operands of kBlk steps.
struct PairOps {
    float2 rv[kBlk], av[kBlk], pi[kBlk];
    float4 da[kBlk];
    double2 b0[kBlk];
    double b11[kBlk];
};

__device__ __forceinline__ int4 ld_cnt4(const int* p) {
    int4 v;
    asm volatile("ld.volatile.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(smem_addr(p))
                 : "memory");
    return v;
}
__device__ __forceinline__ bool reached(int4 v, int4 want) {
    return v.x >= want.x && v.y >= want.y && v.z >= want.z && v.w >= want.w;
}
// Wait until all four counters reach `want` (bounded, as wait_cnt).
__device__ __noinline__ bool wait_cnt4(const int* p, int4 want, int* err) {
    unsigned long long t0 = 0;
    for (uint32_t n = 1;; ++n) {
        if (reached(ld_cnt4(p), want)) return true;
        if ((n & 255) == 0) {
            if (ld_err(err)) return false;
            if (n == 256) {
                t0 = now_ns();
            } else if (now_ns() - t0 > kTimeoutNs) {
                atomicCAS(err, 0, kErrTimeout);
                return false;
            }
        }
    }
}

__device__ __forceinline__ uint64_t ld_pair(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_pair_if(bool ok, uint64_t* p, uint64_t v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t"
                 "@q st.relaxed.gpu.global.b64 [%0], %1;\n\t}" ::"l"(p), "l"(v), "r"((int)ok)
                 : "memory");
}
__device__ __forceinline__ void st_smem_if(bool ok, float2* p, float2 v) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\t@q st.shared.v2.f32 [%0], {%1, %2};\n\t}" ::
                     "r"(smem_addr(p)), "f"(v.x), "f"(v.y), "r"((int)ok)
                 : "memory");
}

// Iteration IT of the CTA's unit on strip k. LAST: the level's last
// iteration. other: the CTA's other sweep runs.
template <int IT, bool LAST>
__device__ __forceinline__ void pair_sweep(const PairArgs& A, PairSmem& M, int k, int c, bool other) {
    const Level L = A.L;
    const int j = threadIdx.x & 31, T = L.w + kLanes - 1;
    const int y = kLanes * k + j;
    const bool rowv = y < L.h, has_next = kLanes * (k + 1) < L.h;
    // Rows without an upper / lower neighbour take their own old value.
    const bool own = (j == 0 && k == 0) || (j == 31 && y == L.h - 1);
    const bool bottom = y == L.h - 1 && j < 31;
    const bool send = j == 31 && has_next, feed = IT == 0 && other && j == 0;
    const long long base = (long long)k * L.Sp * kLanes, cbase = (long long)c * A.pl.n + base;
    uint64_t* mid = A.mid + cbase + j;
    float2* out = A.out + cbase + j;
    uint64_t* bnd = A.bnd + (((long long)IT * A.depth + c) * L.S + k) * L.Sp;
    bool ok = true;
    int4 cv = make_int4(0, 0, 0, 0);
    // Operands of steps s0 .. s0 + kBlk - 1, once they are there.
    auto fetch = [&](int s0, PairOps& o) {
        if (s0 >= T) return;
        // Lane 31 needs the row below at column s - 31. The ring of strip k's
        // first row holds kAux columns for the second iteration on strip
        // k - 1: column x - kAux has left it after that iteration's step
        // x - kAux + 31.
        const int4 want = make_int4(min(s0 + kBlk, L.w),
                                    IT == 0 ? s0 + kBlk - kAux + 31 : min(s0 + kBlk, T - 1) + 1,
                                    min(max(s0 + kBlk - 31, 0), L.w), s0 + kBlk);
        if (!__all_sync(0xffffffffu, reached(cv, want))) ok = ok && wait_cnt4(M.cnt[IT], want, A.err);
        const int slot = (s0 / kPChunk) % kPSlots, sub = s0 & (kPChunk - 1);
        ok = __all_sync(0xffffffffu, ok);
        const PairChunk& C = M.coef[IT][slot];
#pragma unroll
        for (int u = 0; u < kBlk; ++u) {
            const int q = (sub + u) * kLanes + j;
            o.rv[u] = IT == 0 ? M.old[slot][q] : M.rows[((s0 + u + 1) & (kInRows - 1)) * kLanes + j];
            // Lane 0: the strip above at column s. Lane 31: the strip below
            // at column s - 31.
            const float2* a = j != 31 ? &M.up[IT][(s0 + u) & (kAux - 1)]
                              : IT == 0 ? &M.below[slot][sub + u]
                                        : &M.dn1[(s0 + u + kAux - 31) & (kAux - 1)];
            o.av[u] = *a;
            o.da[u] = C.da[q];
            o.b0[u] = C.b0[q];
            o.b11[u] = C.b11[q];
            o.pi[u] = C.pi[q];
        }
        cv = ld_cnt4(M.cnt[IT]);
    };
    float2 p, my;
    auto run = [&](int s0, const PairOps& o) {
#pragma unroll
        for (int u = 0; u < kBlk; ++u) {
            const int s = s0 + u, cur = s - j;
            const float2 dv = shfl_down2(o.rv[u]), uv = shfl_up2(my);
            const float2 a = own ? p : o.av[u];
            const float2 up = j == 0 ? a : uv;
            const float2 dwn = j == 31 ? a : (bottom ? p : dv);
            const float2 rt = cur + 1 < L.w ? o.rv[u] : p;
            const float2 n = fg_pixel(o.pi[u], o.da[u], o.b0[u], o.b11[u], my, rt, up, dwn);
            const bool in = rowv && (unsigned)cur < (unsigned)L.w;
            // Left of the image the lane carries the old value of column 0,
            // which is the left neighbour of column 0.
            my.x = in ? n.x : o.rv[u].x;
            my.y = in ? n.y : o.rv[u].y;
            p = o.rv[u];
            const uint64_t v = pack_fb(n.x, n.y);
            st_pair_if(in, (LAST ? reinterpret_cast<uint64_t*>(out) : mid) + (long long)s * kLanes, v);
            st_pair_if(in && send, bnd + cur, v);
            if (IT == 0) st_smem_if(in && feed, &M.dn1[cur & (kAux - 1)], n);
        }
        put_cnt(&M.done[IT], s0 + kBlk);
        // The first iteration's columns feed the second's row below, whose
        // steps the first must not overrun.
        if (j == 0) {
            volatile int* o2 = &M.cnt[1 - IT][IT == 0 ? kCntDn : kCntRing];
            if (IT == 1) *o2 = s0 + kBlk;
            else if (other) *o2 = min(s0 + kBlk, L.w);
        }
    };
    if (IT == 0) {
        p = A.in[cbase + j];
    } else {
        ok = __all_sync(0xffffffffu, wait_cnt4(M.cnt[IT], make_int4(0, 1, 0, 0), A.err));
        p = M.rows[j];
    }
    my = p;                    // lane 0's column 0 has itself on its left
    PairOps oa, ob;
    fetch(0, oa);
#pragma unroll 1
    for (int s0 = 0; ok && s0 < T; s0 += 2 * kBlk) {
        fetch(s0 + kBlk, ob);
        run(s0, oa);
        if (s0 + kBlk >= T || !ok) break;
        fetch(s0 + 2 * kBlk, oa);
        run(s0 + kBlk, ob);
    }
}

// Bounds a loader's idle rounds. Returns false once it has to give up.
struct Patience {
    uint32_t idle = 0;
    unsigned long long t0 = 0;
    __device__ __forceinline__ bool round(bool moved, int* err) {
        idle = moved ? 0 : idle + 1;
        if (!idle || (idle & 127)) return true;
        bool gave_up = ld_err(err) != 0;
        if (idle == 128) {
            t0 = now_ns();
        } else if (now_ns() - t0 > kTimeoutNs) {
            atomicCAS(err, 0, kErrTimeout);
            gave_up = true;
        }
        return !__any_sync(0xffffffffu, gave_up);
    }
};

// Chunks of both sweeps (strips k and k - 1): coefficients and, for the first
// iteration, starting values and the old row below. The sweeps do not look at
// the barriers themselves (256 cycles a look): a counter tells what landed.
__device__ __forceinline__ void pair_chunks(const PairArgs& A, PairSmem& M, int k, int c, bool it0, bool it1) {
    const Level L = A.L;
    const int j = threadIdx.x & 31, T = L.w + kLanes - 1;
    const int chunks = (T + kPChunk - 1) / kPChunk;
    const float2* dn = A.dn + ((long long)c * L.S + k) * L.Sp;
    int q[2] = {it0 ? 0 : chunks, it1 ? 0 : chunks};      // next chunk to issue
    int landed[2] = {q[0], q[1]};
    Patience P;
    for (bool go = true; go;) {
        if (landed[0] >= chunks && landed[1] >= chunks) return;
        bool moved = false;
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            // Chunk q goes where chunk q - kPSlots was. Its rows exist (Sp is
            // a multiple of 32 and holds every step); the old rows s + 1 may
            // run one row further, into values that no pixel uses.
            if (q[it] < chunks && ld_cnt(&M.done[it]) >= (q[it] - kPSlots + 1) * kPChunk) {
                const int slot = q[it] % kPSlots;
                const long long base = (long long)(k - it) * L.Sp * kLanes + (long long)q[it] * kPChunk * kLanes;
                const long long cbase = (long long)c * A.pl.n + base;
                PairChunk& C = M.coef[it][slot];
                uint64_t* bar = &M.full[it][slot];
                __syncwarp();
                if (j == 0) {
                    fence_proxy_async();
                    mbar_expect_tx(bar, sizeof(PairChunk) +
                                            (it == 0 ? sizeof(M.old[0]) + sizeof(M.below[0]) : 0));
                    bulk_load(C.da, A.pl.da + base, sizeof(C.da), bar);
                    bulk_load(C.b0, A.pl.b0 + base, sizeof(C.b0), bar);
                    bulk_load(C.b11, A.pl.b11 + base, sizeof(C.b11), bar);
                    bulk_load(C.pi, A.pl.pi + cbase, sizeof(C.pi), bar);
                    if (it == 0) {
                        bulk_load(M.old[slot], A.in + cbase + kLanes, sizeof(M.old[0]), bar);
                        bulk_load(M.below[slot], dn + q[it] * kPChunk, sizeof(M.below[0]), bar);
                    }
                }
                __syncwarp();
                ++q[it];
                moved = true;
            }
            if (landed[it] < q[it] &&
                __all_sync(0xffffffffu, mbar_test(&M.full[it][landed[it] % kPSlots],
                                                  (uint32_t)(landed[it] / kPSlots) & 1u))) {
                ++landed[it];
                put_cnt(&M.cnt[it][kCntChunk], landed[it] * kPChunk);
                moved = true;
            }
        }
        go = P.round(moved, A.err);
    }
    // Given up: the CTA does not exit while copies into it are in flight
    // (a bounded wait).
#pragma unroll
    for (int it = 0; it < 2; ++it)
        for (; landed[it] < q[it]; ++landed[it])
            mbar_wait(&M.full[it][landed[it] % kPSlots], (uint32_t)(landed[it] / kPSlots) & 1u);
}

// What other CTAs produce: the border values of the row above strip k (the
// last row of the strip above), and for the second iteration the old rows of
// strip k (row r, lane j: column r - j).
template <int IT>
__device__ __forceinline__ void pair_loader(const PairArgs& A, PairSmem& M, int k, int c) {
    const Level L = A.L;
    const int j = threadIdx.x & 31, T = L.w + kLanes - 1;
    const uint64_t* rows = A.mid + (long long)c * A.pl.n + (long long)k * L.Sp * kLanes + j;
    const uint64_t* up = A.bnd + (((long long)IT * A.depth + c) * L.S + (k > 0 ? k - 1 : 0)) * L.Sp;
    const bool rowv = kLanes * k + j < L.h;
    int r = IT == 1 ? 0 : T, x = k > 0 ? 0 : L.w;      // next row, next column
    Patience P;
    for (bool go = true; go;) {
        if (r >= T && x >= L.w) return;
        bool moved = false;
        const int e = ld_cnt(&M.done[IT]);
        // Row i leaves its ring after step i - 1, column i after step i.
        const int nr = min(min(kRound, T - r), e + kInRows - r);
        const int nx = min(min(kLanes, L.w - x), e + kAux - x);
        uint64_t v[kRound], b = kUnset;
        if (IT == 1) {
#pragma unroll
            for (int i = 0; i < kRound; ++i) {
                v[i] = 0;
                if (i < nr && rowv && (unsigned)(r + i - j) < (unsigned)L.w)
                    v[i] = ld_pair(rows + (long long)(r + i) * kLanes);
            }
        }
        if (j < nx) b = ld_pair(up + x + j);
        if (IT == 1) {
            unsigned have = 0;
#pragma unroll
            for (int i = 0; i < kRound; ++i) have |= i < nr && v[i] != kUnset ? 1u << i : 0u;
            have = __reduce_and_sync(0xffffffffu, have);
            const int got = __ffs(~have) - 1;          // rows from the front
            if (got > 0) {
#pragma unroll
                for (int i = 0; i < kRound; ++i)
                    if (i < got) M.rows[((r + i) & (kInRows - 1)) * kLanes + j] = unpack_fb(v[i]);
                r += got;
                put_cnt(&M.cnt[IT][kCntIn], r);
                moved = true;
            }
        }
        const unsigned miss = __ballot_sync(0xffffffffu, j >= nx || b == kUnset);
        const int m = miss ? __ffs(miss) - 1 : kLanes;
        if (m > 0) {
            if (j < m) M.up[IT][(x + j) & (kAux - 1)] = unpack_fb(b);
            x += m;
            put_cnt(&M.cnt[IT][kCntUp], x);
            moved = true;
        }
        go = P.round(moved, A.err);
    }
}

template <int N_ITER>
__global__ void __launch_bounds__(kPairWarps * kLanes) k_fg_pair(PairArgs A) {
    extern __shared__ __align__(128) unsigned char smem[];
    PairSmem& M = *reinterpret_cast<PairSmem*>(smem);
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        M.unit = atomicAdd(A.ticket, 1);
        for (int i = 0; i < 2; ++i) {
            M.done[i] = 0;
            M.cnt[i][kCntChunk] = 0;
            for (int q = 0; q < kPSlots; ++q) mbar_init(&M.full[i][q], 1);
        }
    }
    __syncthreads();
    const int k = M.unit / A.depth, c = M.unit - k * A.depth;
    const bool it0 = k < A.L.S, it1 = N_ITER == 2 && k > 0;
    if (threadIdx.x == 0) {
        M.cnt[0][kCntUp] = k > 0 ? 0 : kNoWait;
        M.cnt[0][kCntRing] = it1 ? 0 : kNoWait;
        M.cnt[0][kCntDn] = kNoWait;
        M.cnt[1][kCntUp] = k > 1 ? 0 : kNoWait;
        M.cnt[1][kCntIn] = 0;
        M.cnt[1][kCntDn] = it0 ? 0 : kNoWait;        // strip k - 1 is the last one
    }
    __syncthreads();
    if (warp == 0) {
        if (it0) pair_sweep<0, N_ITER == 1>(A, M, k, c, it1);
    } else if (warp == 1) {
        if (it1) pair_sweep<1, true>(A, M, k - 1, c, it0);
    } else if (warp == 2) {
        pair_chunks(A, M, k, c, it0, it1);
    } else if (warp == 3) {
        if (it1) pair_loader<1>(A, M, k - 1, c);
    } else {
        if (it0) pair_loader<0>(A, M, k, c);
    }
}

// ---------------------------------------------------------------------------
// Sweep: all iterations of one level. A CTA holds one warp per colour channel
// of a channel group (at most kGroupMax channels) and works on one unit
// (iteration it, strip k, channel group g) at a time.
// ---------------------------------------------------------------------------

struct SweepArgs {
    Level L;
    int depth, groups, cpg;  // channels, channel groups, channels per group
    const unsigned char* rec;
    ulonglong2* fb;
    float* outF;  // last level only: the final iteration also writes (h, w, depth)
    float* outB;
    int* ticket;
    int* err;
};

__global__ void __launch_bounds__(kLanes * kGroupMax, 1) k_fg_sweep(SweepArgs A) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int s_unit;
    const Level L = A.L;
    const int tid = threadIdx.x, w = tid >> 5, j = tid & 31;
    const int rb = rec_bytes(A.depth);
    const int sbytes = stage_bytes(A.cpg);
    ulonglong2* ring = (ulonglong2*)(smem + 2 * sbytes + w * kWarpRingBytes);
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
    }
    __syncthreads();
    uint32_t phase0 = 0, phase1 = 0;
    const int units = L.n_iter * L.S * A.groups;
    const long long plane = (long long)L.S * L.Sp * kLanes;
    const long long strip = (long long)L.Sp * kLanes;

    for (;;) {
        if (tid == 0) {
            const int u = atomicAdd(A.ticket, 1);
            s_unit = ld_err(A.err) ? units : u;
        }
        __syncthreads();
        const int u = s_unit;
        __syncthreads();
        if (u >= units) break;
        const int g = u % A.groups, ik = u / A.groups;
        const int it = ik / L.S, k = ik - it * L.S;
        const int c0 = g * A.cpg, ng = min(A.cpg, A.depth - c0);
        const unsigned char* rec_k = A.rec + (long long)k * L.Q * rb;
        const uint32_t stage_tx = kBaseBytes + ng * kPIBytes;
        auto stage = [&](int buf, int q) {
            const unsigned char* r = rec_k + (long long)q * rb;
            mbar_expect_tx(&bars[buf], stage_tx);
            bulk_load(smem + buf * sbytes, r, kBaseBytes, &bars[buf]);
            bulk_load(smem + buf * sbytes + kBaseBytes, r + kOffPI + c0 * kPIBytes, ng * kPIBytes,
                      &bars[buf]);
        };
        if (tid == 0) {
            fence_proxy_async();
            for (int b = 0; b < 2 && b < L.Q; ++b) stage(b, b);
        }
        if (w >= ng) {
            // no channel for this warp in this group: keep the phase parities
            // in step with the warps that wait on every chunk
            phase0 ^= (uint32_t)(((L.Q + 1) >> 1) & 1);
            phase1 ^= (uint32_t)((L.Q >> 1) & 1);
            continue;
        }
        const int c = c0 + w;
        ulonglong2* fbc = A.fb + c * plane;
        const int y0 = kLanes * k, y = y0 + j;
        const bool rowv = y < L.h;
        const uint32_t e_old = it, e_new = it + 1;
        const bool has_up = j == 0 && k > 0;
        const bool has_dn = j == 31 && y0 + kLanes < L.h;
        const bool last_out = A.outF != nullptr && it == L.n_iter - 1;
        ulonglong2* row_self = fbc + k * strip + j;
        const ulonglong2* row_up = fbc + (k - 1) * strip + 31;  // used only if has_up
        const ulonglong2* row_dn = fbc + (k + 1) * strip;       // used only if has_dn
        const bool has_aux = has_up || has_dn;
        const uint32_t want_aux = has_up ? e_new : e_old;
        // Step s reads [k][s+1][j] (right-hand value), [k-1][s+31][31] (lane 0)
        // and [k+1][s-31][0] (lane 31): three arithmetic sequences in s.
        const ulonglong2* gR = row_self + kLanes;
        const ulonglong2* gA = has_up ? row_up + 31 * kLanes : (has_dn ? row_dn - 31 * kLanes : row_self);
        const uint32_t ring_lane = smem_addr(ring) + j * 16;

        // Copy the rows step s needs into ring slot s % kRingSlots (zero-filled
        // where the lane has nothing to read). One commit group per step.
        auto issue = [&](int s) {
            const uint32_t slot = ring_lane + (uint32_t)((s & (kRingSlots - 1)) * kRingRow * 16);
            const bool cR = rowv && (unsigned)(s + 1 - j) < (unsigned)L.w;
            const bool cA = has_aux && (unsigned)(s - j) < (unsigned)L.w;
            cp_async16(slot, cR ? gR + (long long)s * kLanes : row_self, cR ? 16u : 0u);
            cp_async16(slot + kLanes * 16, cA ? gA + (long long)s * kLanes : row_self, cA ? 16u : 0u);
            cp_async_commit();
        };
        for (int r = 0; r < kDist; ++r) issue(r);

        float myF = 0.f, myB = 0.f;  // this lane's value from the previous step
        float pF = 0.f, pB = 0.f;    // old value of this lane's current column
        // Lane j first meets its column 0 as the right-hand value of step j-1;
        // for lane 0 that step would be -1, so its column 0 is read here.
        if (j == 0 && rowv) {
            ulonglong2 v = ld_fb(row_self);
            if (!has_epoch(v, e_old)) v = poll_epoch(row_self, e_old, A.err);
            pF = value_of(v.x);
            pB = value_of(v.y);
        }
        const int nthr = kLanes * ng;
        for (int q = 0; q < L.Q; ++q) {
            uint64_t* bar = &bars[q & 1];
            const uint32_t ph = (q & 1) ? phase1 : phase0;
            if (!mbar_wait(bar, ph)) atomicCAS(A.err, 0, kErrStage);
            if (q & 1) phase1 ^= 1u; else phase0 ^= 1u;
            const unsigned char* cb = smem + (q & 1) * sbytes;
            // the last step with work is w + 30 (lane 31 at column w - 1)
            const int t_end = min(kChunk, L.w + kLanes - 1 - kChunk * q);
// not unrolled: the rolled loop measured 33 % faster than unroll 4
#pragma unroll 1
            for (int t = 0; t < t_end; ++t) {
                const int s = kChunk * q + t;
                const int cur = s - j;
                cp_async_wait<kDist - 1>();
                const ulonglong2* slot = ring + (s & (kRingSlots - 1)) * kRingRow;
                ulonglong2 Rv = slot[j];
                ulonglong2 Av = slot[kLanes + j];
                // the slot refilled now was read at step s - 1
                issue(s + kDist);
                const bool inCol = (unsigned)cur < (unsigned)L.w;
                const bool needR = rowv && (unsigned)(cur + 1) < (unsigned)L.w;
                const bool needA = has_aux && inCol;
                const bool okR = !needR || has_epoch(Rv, e_old);
                const bool okA = !needA || has_epoch(Av, want_aux);
                if (!__all_sync(0xffffffffu, okR && okA)) {
                    if (!okR) Rv = poll_epoch(gR + (long long)s * kLanes, e_old, A.err);
                    if (!okA) Av = poll_epoch(gA + (long long)s * kLanes, want_aux, A.err);
                }
                const float rF = value_of(Rv.x), rB = value_of(Rv.y);
                const float aF = value_of(Av.x), aB = value_of(Av.y);
                const float uF = __shfl_up_sync(0xffffffffu, myF, 1);
                const float uB = __shfl_up_sync(0xffffffffu, myB, 1);
                const float dF = __shfl_down_sync(0xffffffffu, rF, 1);
                const float dB = __shfl_down_sync(0xffffffffu, rB, 1);
                const bool first = cur == 0, rin = cur + 1 < L.w;
                const bool top = y == 0, bottom = y == L.h - 1;
                const float Fl = first ? pF : myF, Bl = first ? pB : myB;
                const float Fr = rin ? rF : pF, Br = rin ? rB : pB;
                const float Fu = top ? pF : (j == 0 ? aF : uF);
                const float Bu = top ? pB : (j == 0 ? aB : uB);
                const float Fd = bottom ? pF : (j == 31 ? aF : dF);
                const float Bd = bottom ? pB : (j == 31 ? aB : dB);
                const int e = (t << 5) | j;
                const float4 da = *(const float4*)(cb + kOffDa + e * 16);
                const double2 b0 = *(const double2*)(cb + kOffB0 + e * 16);
                const double b11 = *(const double*)(cb + kOffB11 + e * 8);
                const float2 pI = *(const float2*)(cb + kOffPI + w * kPIBytes + e * 8);
                float f0 = pI.x, f1 = pI.y;
                f0 = __fadd_rn(f0, __fmul_rn(da.x, Fl));
                f1 = __fadd_rn(f1, __fmul_rn(da.x, Bl));
                f0 = __fadd_rn(f0, __fmul_rn(da.y, Fr));
                f1 = __fadd_rn(f1, __fmul_rn(da.y, Br));
                f0 = __fadd_rn(f0, __fmul_rn(da.z, Fu));
                f1 = __fadd_rn(f1, __fmul_rn(da.z, Bu));
                f0 = __fadd_rn(f0, __fmul_rn(da.w, Fd));
                f1 = __fadd_rn(f1, __fmul_rn(da.w, Bd));
                double Fc = __dadd_rn(__dmul_rn(b0.x, (double)f0), __dmul_rn(b0.y, (double)f1));
                double Bc = __dadd_rn(__dmul_rn(b0.y, (double)f0), __dmul_rn(b11, (double)f1));
                // max(0.0, min(1.0, v)) with Python's argument order
                Fc = Fc < 1.0 ? Fc : 1.0;
                Fc = Fc > 0.0 ? Fc : 0.0;
                Bc = Bc < 1.0 ? Bc : 1.0;
                Bc = Bc > 0.0 ? Bc : 0.0;
                const float nF = __double2float_rn(Fc), nB = __double2float_rn(Bc);
                if (rowv && inCol) {
                    st_fb(row_self + (long long)s * kLanes, pack(nF, e_new), pack(nB, e_new));
                    if (last_out) {
                        const long long o = ((long long)y * L.w + cur) * A.depth + c;
                        A.outF[o] = nF;
                        if (A.outB) A.outB[o] = nB;
                    }
                }
                // (garbage in lanes outside the image; nothing reads it there)
                myF = nF;
                myB = nB;
                pF = rF;
                pB = rB;
            }
            // every active warp is done with this buffer: refill it with chunk q + 2
            bar_sync1(nthr);
            if (tid == 0 && q + 2 < L.Q) {
                fence_proxy_async();
                stage(q & 1, q + 2);
            }
        }
        cp_async_wait<0>();
    }
}

// Result images (h, w, depth) from the last level's diagonal layout. A CTA
// moves 32 columns of a strip: the diagonal rows that hold them are read
// whole, and leave through shared memory as contiguous image rows.
__global__ void __launch_bounds__(256) k_fg_output(Level L, int depth, const void* __restrict__ fb,
                                                   float* __restrict__ outF, float* __restrict__ outB) {
    __shared__ float2 tile[kLanes][kLanes + 1];
    const int k = blockIdx.y, x0 = blockIdx.x * kLanes, j = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long plane = (long long)L.S * L.Sp * kLanes, base = (long long)k * L.Sp * kLanes;
    for (int c = 0; c < depth; ++c) {
        for (int r = warp; r < 2 * kLanes - 1; r += 8) {
            const int x = r - j;                               // column within the tile
            if (x < 0 || x >= kLanes || x0 + x >= L.w || kLanes * k + j >= L.h) continue;
            const long long i = c * plane + base + (long long)(x0 + r) * kLanes + j;
            if (L.tagged) {
                const ulonglong2 u = static_cast<const ulonglong2*>(fb)[i];
                tile[j][x] = make_float2(value_of(u.x), value_of(u.y));
            } else {
                tile[j][x] = static_cast<const float2*>(fb)[i];
            }
        }
        __syncthreads();
        for (int r = warp; r < kLanes; r += 8) {
            const int y = kLanes * k + r, x = x0 + j;
            if (y < L.h && x < L.w) {
                const long long o = ((long long)y * L.w + x) * depth + c;
                outF[o] = tile[r][j].x;
                if (outB) outB[o] = tile[r][j].y;
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// Level sizes of estimate_foreground_ml.py:101-105 (glibc pow and log2, ties
// of round() to even). Returns the level count, or -1 for a 1x1 image (the
// reference divides by zero there).
static int plan_levels(int h0, int w0, int n_small, int n_big, int small_size, Level* out) {
    const int m = std::max(h0, w0);
    const int n = (int)std::ceil(std::log2((double)m));
    if (n == 0) return -1;
    if (n + 1 > kMaxLevels) return -2;
    for (int i = 0; i <= n; ++i) {
        const double e = (double)i / (double)n;
        Level& L = out[i];
        L.w = (int)std::nearbyint(std::pow((double)w0, e));
        L.h = (int)std::nearbyint(std::pow((double)h0, e));
        L.S = (L.h + kLanes - 1) / kLanes;
        L.Q = (L.w + kLanes - 1 + kChunk - 1) / kChunk;
        L.Sp = L.Q * kChunk;
        L.n_iter = (L.w <= small_size && L.h <= small_size) ? n_small : n_big;
        // One or two iterations: k_fg_pair. More are in flight together only
        // in k_fg_sweep (each adds about 40 steps to a level's chain there, a
        // whole pass over it in k_fg_pair).
        L.tagged = L.n_iter > 2;
    }
    return n + 1;
}

static long long align256(long long v) { return (v + 255) & ~255LL; }

struct Layout {
    long long hdr, part, seed, fb0, fb1, bnd, dn, rec, total;
};

static Layout layout(int h0, int w0, int depth) {
    const int S = (h0 + kLanes - 1) / kLanes;
    const int Q = (w0 + kLanes - 1 + kChunk - 1) / kChunk;
    const long long fb = (long long)depth * S * Q * kChunk * kLanes * 16;
    Layout l;
    l.hdr = 0;
    l.part = 1024;
    l.seed = l.part + align256((long long)kMeanBlocks * kMeanValues * 8);
    l.fb0 = l.seed + 256;
    l.fb1 = l.fb0 + align256(fb);
    l.bnd = l.fb1 + align256(fb);
    l.dn = l.bnd + align256((long long)2 * depth * S * Q * kChunk * 8);
    l.rec = l.dn + align256((long long)depth * S * Q * kChunk * 8);
    l.total = l.rec + align256((long long)S * Q * rec_bytes(depth));
    return l;
}

// Self-test of the bounded poll: one thread waits with poll_epoch for epoch
// 1 in a word that holds epoch 0 and that nothing writes, with a deadline of
// timeout_ns. The poll must give up and leave kErrTimeout in *err.
__global__ void k_selftest_poll(const ulonglong2* word, int* err, unsigned long long timeout_ns) {
    if (threadIdx.x == 0 && blockIdx.x == 0) (void)poll_epoch(word, 1u, err, timeout_ns);
}

}  // namespace fg
}  // namespace pmb

using namespace pmb::fg;

// scratch: 64 bytes of device memory. Returns 0 and sets *timed_out (1 if
// the poll gave up and reported it), or a CUDA error code.
int pmb_launch_selftest_poll(void* scratch, unsigned long long timeout_ns, int* timed_out,
                             cudaStream_t st) {
    ulonglong2* word = static_cast<ulonglong2*>(scratch);
    int* err = reinterpret_cast<int*>(static_cast<char*>(scratch) + 32);
    cudaError_t e = cudaMemsetAsync(scratch, 0, 64, st);
    if (e != cudaSuccess) return (int)e;
    k_selftest_poll<<<1, 32, 0, st>>>(word, err, timeout_ns);
    int h = 0;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    *timed_out = h == kErrTimeout ? 1 : 0;
    return 0;
}

int64_t pmb_launch_fg_workspace(int h, int w, int depth) {
    if (h <= 0 || w <= 0 || depth < 1 || depth > kMaxDepth) return -1;
    return layout(h, w, depth).total;
}

int pmb_launch_fg_levels(int h, int w, int n_small, int n_big, int small_size, int* hw, int max_levels) {
    Level lv[kMaxLevels];
    const int n = plan_levels(h, w, n_small, n_big, small_size, lv);
    if (n < 0) return n;
    for (int i = 0; i < n && i < max_levels; ++i) {
        hw[2 * i] = lv[i].h;
        hw[2 * i + 1] = lv[i].w;
    }
    return n;
}

// Returns 0, -1 (1x1 image), -2 (bad arguments), -3 (workspace too small) or
// a positive CUDA error code.
int pmb_launch_fg(const float* image, const float* alpha, int h0, int w0, int depth, float reg,
                  int n_small, int n_big, int small_size, float gw, const float* seed_in,
                  float* outF, float* outB, void* workspace, int64_t ws_bytes, cudaStream_t st) {
    if (!image || !alpha || !outF || !workspace || h0 <= 0 || w0 <= 0 || h0 > kMaxSide ||
        w0 > kMaxSide || depth < 1 || depth > kMaxDepth || n_small < 0 || n_big < 0)
        return -2;
    Level lv[kMaxLevels];
    const int nl = plan_levels(h0, w0, n_small, n_big, small_size, lv);
    if (nl == -1) return -1;
    if (nl < 0) return -2;
    const Layout l = layout(h0, w0, depth);
    if (ws_bytes < l.total) return -3;
    unsigned char* ws = (unsigned char*)workspace;
    int* hdr = (int*)(ws + l.hdr);  // [0] error word, [1 + level] ticket counters
    double* part = (double*)(ws + l.part);
    float* seed = (float*)(ws + l.seed);
    unsigned char* fbs[2] = {ws + l.fb0, ws + l.fb1};
    const long long half = (l.fb1 - l.fb0) / 512 * 256;    // a level's float2 values, twice in a region
    unsigned char* rec = ws + l.rec;

    int dev = 0, num_sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (num_sms <= 0) num_sms = 148;
    const int groups = (depth + kGroupMax - 1) / kGroupMax;
    const int cpg = (depth + groups - 1) / groups;
    const int sweep_smem = 2 * stage_bytes(cpg) + cpg * kWarpRingBytes;
    cudaError_t e = cudaFuncSetAttribute(k_fg_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         2 * stage_bytes(kGroupMax) + kGroupMax * kWarpRingBytes);
    if (e != cudaSuccess) return (int)e;
    e = cudaMemsetAsync(hdr, 0, 1024, st);
    if (e != cudaSuccess) return (int)e;
    if (!seed_in) {
        const long long n = (long long)h0 * w0;
        k_fg_mean_partial<<<kMeanBlocks, kMeanThreads, 0, st>>>(image, alpha, n, depth, part);
        k_fg_mean_final<<<1, 32 * kMeanValues, 0, st>>>(part, kMeanBlocks, depth, seed);
        seed_in = seed;
    }
    // The first levels in one launch.
    SmallArgs SA{};
    int small_iters = 1;
    while (SA.n < nl && SA.n < kSmallLevels && lv[SA.n].h <= kSmallSide && lv[SA.n].w <= kSmallSide &&
           lv[SA.n].n_iter <= kSmallIters) {
        lv[SA.n].tagged = 0;
        SA.lv[SA.n] = lv[SA.n];
        small_iters = std::max(small_iters, lv[SA.n].n_iter);
        ++SA.n;
    }
    // Region (0 or 1) and offset of the previous level's result.
    int prev = 1;
    if (SA.n > 0) {
        SA.image = image;
        SA.alpha = alpha;
        SA.h0 = h0;
        SA.w0 = w0;
        SA.depth = depth;
        SA.reg = reg;
        SA.gw = gw;
        SA.seed = seed_in;
        SA.out = (float2*)fbs[1];
        SA.err = hdr;
        e = cudaFuncSetAttribute(k_fg_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallSmem));
        if (e != cudaSuccess) return (int)e;
        // eight warps at least: they share the preparation of a level
        k_fg_small<<<depth, kLanes * std::max(small_iters, 8), sizeof(SmallSmem), st>>>(SA);
        if (SA.n == nl) {
            k_fg_output<<<dim3((w0 + kLanes - 1) / kLanes, lv[nl - 1].S), 256, 0, st>>>(lv[nl - 1], depth, fbs[1],
                                                                                      outF, outB);
        }
    }
    Level none{};
    for (int i = SA.n; i < nl; ++i) {
        const Level& L = lv[i];
        const bool last = i == nl - 1;
        unsigned char* fresh = fbs[1 - prev];
        PrepArgs P;
        P.image = image;
        P.alpha = alpha;
        P.h0 = h0;
        P.w0 = w0;
        P.depth = depth;
        P.reg = reg;
        P.gw = gw;
        P.L = L;
        P.P = i > 0 ? lv[i - 1] : none;
        P.fb_prev = fbs[prev];
        P.seed = seed_in;
        P.rec = rec;
        P.fb = fresh;
        P.mid = (uint64_t*)(fresh + half);
        P.bnd = (uint64_t*)(ws + l.bnd);
        P.dn = (float2*)(ws + l.dn);
        const dim3 pgrid((L.Sp * kLanes + 255) / 256, L.S);
        k_fg_prep<<<pgrid, 256, 0, st>>>(P);
        if (L.n_iter > 0 && !L.tagged) {
            PairArgs S;
            S.L = L;
            S.depth = depth;
            S.pl = planes_of(rec, L);
            S.in = (const float2*)fresh;
            S.mid = P.mid;
            S.out = (float2*)fbs[prev];          // the previous level's values are read by now
            S.bnd = P.bnd;
            S.dn = P.dn;
            S.ticket = hdr + 1 + i;
            S.err = hdr;
            auto kernel = L.n_iter == 2 ? k_fg_pair<2> : k_fg_pair<1>;
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PairSmem));
            if (e != cudaSuccess) return (int)e;
            kernel<<<(L.S + (L.n_iter == 2 ? 1 : 0)) * depth, kPairWarps * kLanes, sizeof(PairSmem), st>>>(S);
            if (last)
                k_fg_output<<<dim3((w0 + kLanes - 1) / kLanes, L.S), 256, 0, st>>>(L, depth, S.out, outF, outB);
        } else if (L.n_iter > 0) {
            SweepArgs S;
            S.L = L;
            S.depth = depth;
            S.groups = groups;
            S.cpg = cpg;
            S.rec = rec;
            S.fb = (ulonglong2*)fresh;
            S.outF = last ? outF : nullptr;
            S.outB = last ? outB : nullptr;
            S.ticket = hdr + 1 + i;
            S.err = hdr;
            const int units = L.n_iter * L.S * groups;
            const int grid = std::min(units, num_sms);
            k_fg_sweep<<<grid, kLanes * cpg, sweep_smem, st>>>(S);
            prev = 1 - prev;
        } else {
            if (last) {
                k_fg_output<<<dim3((w0 + kLanes - 1) / kLanes, L.S), 256, 0, st>>>(L, depth, fresh, outF, outB);
            }
            prev = 1 - prev;
        }
    }
    e = cudaGetLastError();
    return e == cudaSuccess ? 0 : (int)e;
}

// Error word of the last run in `workspace` (synchronises the stream).
int pmb_launch_fg_status(void* workspace, cudaStream_t st, int* status) {
    int v = 0;
    cudaError_t e = cudaMemcpyAsync(&v, workspace, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return (int)e;
    *status = v;
    return 0;
}
