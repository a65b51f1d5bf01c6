// Learned initial-partition proposal: shared declarations of the network kernels (mpnn_kernels.cu) and the
// C-ABI (mpnn_cabi.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "batch.cuh"

namespace dmolp {
namespace mpnn {

constexpr int kIn = 16, kHidden = 64, kOut = 16;
constexpr int kAnchors = 8;
constexpr int kTMax = 96;
constexpr float kMargin = 1.0f;
constexpr float kPFloor = 1e-30f;
// layer l: [K_l x N_l] weights + N_l biases, K_l = 2 * (input width)
constexpr int kK[3] = {2 * kIn, 2 * kHidden, 2 * kHidden};
constexpr int kN[3] = {kHidden, kHidden, kOut};
constexpr int kNumParams = 2 * kIn * kHidden + kHidden + 2 * kHidden * kHidden + kHidden + 2 * kHidden * kOut + kOut;

enum GemmKind { kFwd = 0, kBwdData = 1, kBwdWeight = 2 };

struct GemmArgs {
    int kind;
    int rows;        // vertices
    int K;           // kFwd / kBwdData: reduction length (multiple of 16)
    int nb;          // valid B rows (kFwd / kBwdData) or valid output columns
    int m_valid;     // kBwdWeight: valid rows of dW
    int chunk;       // kBwdWeight: vertices per work item (multiple of the K tile)
    const __nv_bfloat16 *A;
    int lda;
    const __nv_bfloat16 *B;
    int ldb;
    const float *bias;
    int relu;
    __nv_bfloat16 *out_bf16;
    int ldo;
    float *out_f32;
    int ldo32;
    const int64_t *off;  // kBwdData: columns >= kHidden are divided by the row's degree
    float *out_w;
    int *err;
    uint32_t polls;  // polls of the MMA completion barrier before the GEMM gives up (then: err, TMEM freed)
};

// One launch of the tensor-core GEMM, N = n: row kinds with (n, K) = (64, 32), (64, 128), (16, 128), (128, 16) or
// (128, 64), the weight gradient with n = 64 or 16.
void gemm(const GemmArgs &g, int n, int num_sms, cudaStream_t s);

void agg_fwd(const batch::View &b, __nv_bfloat16 *buf, int C);
void agg_bwd(const batch::View &b, const float *dC, const __nv_bfloat16 *Hbuf, int ldh, __nv_bfloat16 *G, float *db);
void loss(const int64_t *off, const int32_t *col, int nv, const float *Z, const int32_t *target, double inv_arcs,
          __nv_bfloat16 *G, float *db, double *loss_sum, int num_sms, cudaStream_t s);
void grad_out(const float *dZ, int nv, __nv_bfloat16 *G, float *db, int num_sms, cudaStream_t s);
void adam(float *p, const float *g, float *m, float *v, int n, float lr, int step, cudaStream_t s);
void cast_weights(const float *params, __nv_bfloat16 *const W[3], __nv_bfloat16 *const Wt[3], cudaStream_t s);

// A work unit of the walk: n <= kChunkV consecutive vertices of one graph, or (n = 0) the long row of v0.
constexpr int kChunkV = 256;
struct Chunk {
    int v0, n, inst;
};

// A vertex's row and its distance to the nearest anchor so far.
struct __align__(16) SearchRow {
    int64_t start;
    int len, dist;
};

constexpr size_t kFeatSharedBytes = 1024;

struct FeatWork {
    const int64_t *off;
    const int32_t *col;
    const batch::Inst *inst;
    int ninst;
    int nv;
    int32_t *vinst;                           // [nv]
    SearchRow *row, *front0, *front1, *huge;  // [nv] search state; frontiers and long rows in per-graph slices
    int *next;                                // the teams' queue
    int32_t *anchor;                          // [kAnchors * ninst]
    int32_t *ecc;                             // [ninst]
    Chunk *chunks;                            // [nv / kChunkV + ninst + the batch's long rows]
    float *P0, *Q0, *P1, *Q1;                 // [nv * 8]
    double *stats;                            // [ninst * 16]
    void *shared;                             // [kFeatSharedBytes] counters of the searches' largest teams
    int *err;                                 // set by a wait that gave up after `polls` polls
    uint32_t polls;
    float *Xf;                                // [nv * 16] features before rounding
    __nv_bfloat16 *X;                         // [nv * ldx] bf16 input of layer 1
    int ldx;
};
int features(const FeatWork &w, const batch::View &b, cudaStream_t s);  // returns a CUDA error code (0 = ok)
void features_to_input(const float *Xf, int nv, __nv_bfloat16 *X, int ldx, int num_sms, cudaStream_t s);

// The decoder's records: kDecRecord sums per segment of a part that splits, all but a part's last of at least kDecSeg
// vertices, at most kDecSplits such parts at once.  A graph's records start at decode_record of its first vertex and its index.
constexpr int kDecSeg = 128, kDecRecord = 36, kDecSplits = batch::kBatchMaxK / 2;
__host__ __device__ __forceinline__ size_t decode_record(int64_t vbase, int inst) {
    return (size_t)(vbase / kDecSeg) + (size_t)kDecSplits * inst;
}

struct DecodeWork {
    const batch::Inst *inst;
    const float *Z;     // [nv * 16] proposal coordinates (first 8 columns used)
    uint64_t *key;      // [nv] work
    double *rec;        // [decode_record(nv, ninst) * kDecRecord] work
    int32_t *label;
    int32_t *l0, *l1;   // [nv] each: work
    int32_t *status;    // [ninst]
    int *next;
};
// The graphs of `order` (host and device copies, largest first).  Returns a CUDA error code (0 = ok).
int decode(const DecodeWork &w, const std::vector<int32_t> &order, const int32_t *d_order, const batch::View &b,
           cudaStream_t s);
void coords(const float *Xf, const float *Z, int nv, float *P, int num_sms, cudaStream_t s);
void gate_scores(const float *Z, const int32_t *vinst, int nv, double *score, int num_sms, cudaStream_t s);
void gate_grad(const float *g, const int32_t *vinst, int nv, float *dZ, int num_sms, cudaStream_t s);

}  // namespace mpnn
}  // namespace dmolp
