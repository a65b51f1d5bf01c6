// Batched LP: device-side instance table and kernel arguments (batch_kernels.cu), used by batch_cabi.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "../../include/dmolp_b200.h"
#include "common.cuh"

namespace dmolp {

// The reference's hub list of a graph from its per-vertex degrees (src/phase1/init.cpp:139-177), as the
// single-graph path computes it (dmolp_cabi.cu).
std::vector<int> hubs_of(const std::vector<int32_t> &degree);

namespace batch {

constexpr int kBatchMaxK = DMOLP_BATCH_MAX_K;
constexpr int kLongRow = 256;      // the per-vertex network kernels give longer rows a block each
constexpr int kStampStride = 512;  // > the longest run (kMaxIter iterations)

struct Inst {
    int64_t vbase;   // first vertex of the instance in the union graph
    int64_t narcs;   // arcs of the instance
    int32_t nv, k;
    int32_t maxdeg, ibits, dbits, symmetric;
    int64_t cbase;    // its first kept label count
    int32_t cstride;  // 16-bit counts per vertex (min(k, 32) rounded up to 8); 0 = no kept counts
};

struct Out {
    long long edge_cut, te, arcs, visits;
    int iterations, stop_reason, status, changes;
};

struct Args {
    const int64_t *off;
    const int32_t *col;
    int32_t *label, *newlab, *cstamp;
    int32_t *ndiff;  // neighbours with another label, exact at every iteration start
    int32_t *l_bnd, *l_win0, *l_win1;  // per-instance slices at vbase
    uint64_t *rec0, *rec1;             // selection records, per-instance slices at vbase
    uint16_t *cnt;                     // kept label counts, per-instance slices at cbase (null: no graph has any)
    const Inst *inst;
    const int32_t *order;
    int ninst;
    int *next, *stamp_base;
    Out *out;
    long long *counts;  // [ninst][2 * kBatchMaxK]: vertex counts, intra-part edges
    const double *logtab, *ratiotab;
    int mode, iters, cap;
};

// Batched phase 1 (batch_p1.cu).
struct P1Out {
    int nseeds_found, rounds;
    unsigned long long te;
};

struct P1Args {
    const int64_t *off;
    const int32_t *col;
    int32_t *label;
    const Inst *inst;
    int *next;
    const int32_t *hubs;    // per graph, local ids in the reference's hub order (descending degree)
    const int64_t *hstart;  // [ninst + 1]
    const int32_t *first;   // [ninst] first seed (local id)
    uint8_t *cov;
    int32_t *claim;
    int32_t *l_front0, *l_front1, *l_sel;  // per-graph slices at vbase
    uint64_t *rec0, *rec1;                 // selection records, per-graph slices at vbase
    int32_t *seeds_out;                    // [ninst][kBatchMaxK]
    P1Out *out;
    int theta;
};

// Teams: the batch's graphs, in `order` (largest first), are run by clusters of 16, 8, 4 and 2 CTAs and by
// single CTAs; n[j] graphs by teams of kMaxTeam >> j.
constexpr int kMaxTeam = 16;
constexpr int kTeamClasses = 5;
struct TeamPlan {
    int n[kTeamClasses];
};

// Side streams on which the classes of a plan run next to each other (the plan's first class runs on the
// stream itself): open() makes them wait for what is on the stream, close() makes the stream wait for them.
struct Fork {
    cudaStream_t side[kTeamClasses - 1];
    cudaEvent_t begin, end[kTeamClasses - 1];
    static int lead(const TeamPlan &p) {
        int j = 0;
        while (j < kTeamClasses - 1 && p.n[j] == 0) ++j;
        return j;
    }
    cudaStream_t stream(const TeamPlan &p, int j, cudaStream_t s) const { return j == lead(p) ? s : side[j - 1]; }
    void open(const TeamPlan &p, cudaStream_t s) const {
        bool first = true;
        for (int j = lead(p) + 1; j < kTeamClasses; ++j) {
            if (p.n[j] == 0) continue;
            if (first) cudaEventRecord(begin, s);
            first = false;
            cudaStreamWaitEvent(side[j - 1], begin, 0);
        }
    }
    void close(const TeamPlan &p, cudaStream_t s) const {
        for (int j = lead(p) + 1; j < kTeamClasses; ++j) {
            if (p.n[j] == 0) continue;
            cudaEventRecord(end[j - 1], side[j - 1]);
            cudaStreamWaitEvent(s, end[j - 1], 0);
        }
    }
};

// What the other device modules (the learned proposal) need of a resident batch.
struct View {
    const int64_t *off;
    const int32_t *col;
    int32_t *label;
    const Inst *inst;
    const int32_t *order;
    const int32_t *longrow;  // [nlong] vertices of more than kLongRow arcs
    int ninst, nlong;
    int64_t nv, narcs;
    cudaStream_t stream;
    int num_sms, device;
    const std::vector<Inst> *h_inst;      // the same table and order on the host
    const std::vector<int32_t> *h_order;
    const std::vector<int32_t> *h_longrow;  // ascending
    const Fork *fork;
};
bool view(dmolp_batch *b, View *v);  // false when nothing is uploaded

// CTAs per graph of `order` (batch_cabi.cu).
TeamPlan team_sizes(const std::vector<Inst> &inst, const std::vector<int32_t> &order, int slots, int nt, int most);

// Whether clusters of c CTAs of the kernel can run, and how many at once.
template <typename K>
bool max_clusters(K kernel, int c, int nt, int *n, size_t smem = 0) {
    if (c > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)c;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3((unsigned)nt);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(n, kernel, &cfg) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

// n clusters of c CTAs (max_clusters has been asked for this kernel and c).
template <typename K, typename... A>
cudaError_t launch_cluster_smem(K kernel, int n, int c, int nt, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)c;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(n * c));
    cfg.blockDim = dim3((unsigned)nt);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename K, typename... A>
cudaError_t launch_cluster(K kernel, int n, int c, int nt, cudaStream_t s, A... args) {
    return launch_cluster_smem(kernel, n, c, nt, 0, s, args...);
}

int p1_threads();
int p1_max_team();
void launch_p1(const P1Args &a, const int32_t *order, int grid, const TeamPlan &plan, const Fork &f, cudaStream_t s);

int occupancy(int nt, int td);
int max_team(int nt, int td);  // the largest cluster the device can run, 1 if none
bool launch(const Args &a, int nt, int td, int grid, const TeamPlan &plan, const Fork &f, cudaStream_t s);
void prepare(const int64_t *off, int32_t *col, Inst *inst, int ninst, int64_t nv, int64_t narcs, int *err,
             int32_t *longrow, int *nlong, int grid, cudaStream_t s);

}  // namespace batch
}  // namespace dmolp
