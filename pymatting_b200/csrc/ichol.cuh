// Launch interface of the incomplete-Cholesky kernels (ichol.cu).
#pragma once

#include "pm_common.cuh"

namespace pmb {

// Streamed solves: chunk limits, stages in flight and the largest system
// whose x fits in shared memory beside the stages.
constexpr int kStreamRowsMax = 64;
constexpr int kStreamEntsMax = 512;
constexpr int kStreamStages = 8;
constexpr int64_t kStreamMaxRows = 20000;
constexpr uint32_t kStreamSpinLimit = 1u << 24;

// Records of a chunk block: its head, then one per row.
struct StreamHead {
    int64_t next_off;      // byte offset of the chunk kStreamStages later
    int next_bytes;        // its size (0: none)
    int rows, ents;        // this chunk
    int pad[3];
};
struct StreamRow {
    int row, start, count;
    int fast;              // inv serves the quotient (root_range)
    double diag, inv;      // L_ii and its reciprocal
};
static_assert(sizeof(StreamHead) == 32 && sizeof(StreamRow) == 32, "chunk records are 32 bytes");

// Offsets and sizes of the first kStreamStages chunk blocks (later ones are
// named by the block kStreamStages before them).
struct StreamFirst {
    int64_t off[kStreamStages];
    int bytes[kStreamStages];
};
// Host-built packing plan: one record per row of each sweep, one per chunk.
struct StreamPackRow {
    int64_t chunk_off;   // byte offset of the row's chunk block
    int64_t src;         // first entry in the row view (forward) or column of L (backward)
    int row, slot, start, count;
    int rows, ents;      // of the row's chunk
    int backward, pad;
};
struct StreamPackChunk {
    int64_t off;
    int bytes, rows, ents, used;   // used: entries before padding
};

size_t ichol_stream_smem(int64_t n);
void ichol_launch_stream_pack(int nrec, const StreamPackRow* recs, int nchunks,
                              const StreamPackChunk* chunks, const int64_t* Rc, const double* Rv,
                              const int64_t* Lr, const double* Lv, const int64_t* Lp,
                              unsigned char* blob, cudaStream_t s);
void ichol_launch_solve_stream(int64_t n, int total, const StreamFirst& first,
                               const unsigned char* blob, const double* b, double* x,
                               const InstState* st, uint32_t limit, cudaStream_t s);

void ichol_launch_init(int64_t n, const int64_t* Ap, const int64_t* Ar, const double* Av,
                       double shift, double* d, double* rsum, int* level, unsigned long long* band,
                       cudaStream_t s);
// Result of the pipelined kernel when a wait ran out: the factor is made by
// ichol_launch_factor.
constexpr int64_t kIcholRetry = -100;
// ... and when the columns are long: ichol_launch_factor_cluster makes it.
constexpr int64_t kIcholDense = -101;
constexpr uint32_t kPipeSpinLimit = 1u << 22;
// Kernel that made a factor: the front in global memory (also after a retry),
// the pipeline, the front in a cluster's shared memory.
enum : int { kIcholByGlobal = 0, kIcholByPipe = 1, kIcholByCluster = 2, kIcholByRetry = 3 };
constexpr int64_t kPipeMinW = 8;      // rows of its ring (narrower bands are padded)
bool ichol_launch_factor_pipe(int64_t n, int64_t W, const int64_t* Ap, const int64_t* Ar,
                              const double* Av, const double* d, const double* rsum, int* level,
                              int64_t* Lp, int64_t* Lr, double* Lv, double* list, uint16_t* offs, int64_t cap,
                              double discard, int64_t max_nnz, double rel, int diag_keep,
                              int64_t* result, uint32_t limit, int look_cols, int64_t look_end,
                              int64_t dense_nnz, cudaStream_t s);
// The front in a cluster's shared memory (ichol_cluster.cu). False: not launched.
bool ichol_launch_factor_cluster(int64_t n, int64_t W, const int64_t* Ap, const int64_t* Ar,
                                 const double* Av, const double* d, const double* rsum, int* level,
                                 int64_t* Lp, int64_t* Lr, double* Lv, int64_t cap, double discard,
                                 int64_t max_nnz, double rel, int diag_keep, int64_t* result,
                                 cudaStream_t s);
int64_t ichol_dense_columns(int64_t W);
// The global-front kernel: bands that the pipelined kernel does not take.
void ichol_launch_factor(int64_t n, int64_t W, const int64_t* Ap, const int64_t* Ar,
                        const double* Av, double* d, const double* rsum, int* level, double* F,
                        uint8_t* pat, int* cand, double* keptv, int64_t* kepti, int64_t* Lp,
                        int64_t* Lr, double* Lv, int64_t cap, double discard, int64_t max_nnz,
                        double rel, int diag_keep, int64_t* result, cudaStream_t s);
void ichol_launch_levels(int64_t n, const int* level, int64_t* cnt, int* maxlevel, cudaStream_t s);
void ichol_launch_level_scatter(int64_t n, const int* level, int64_t* fill, int* order,
                                const int64_t* lptr, int nlevels, cudaStream_t s);
void ichol_launch_rows(int64_t n, const int64_t* Lp, const int64_t* Lr, const double* Lv,
                       int64_t* rcnt, cudaStream_t s);
void ichol_launch_row_fill(int64_t n, const int64_t* Lp, const int64_t* Lr, const double* Lv,
                           int64_t* rfill, int64_t* Rc, double* Rv, const int64_t* Rp,
                           cudaStream_t s);
// CTAs of the cluster whose shared memory the band front of W rows fills; 0 if
// it has no room there.
int ichol_cluster_size(int64_t W);
void ichol_prepare();
void ichol_launch_solve(int64_t n, int nlevels, const int64_t* lptr, const int* order,
                        const int64_t* Lp, const int64_t* Lr, const double* Lv, const int64_t* Rp,
                        const int64_t* Rc, const double* Rv, const double* b, double* x,
                        const InstState* st, cudaStream_t s);

}  // namespace pmb
