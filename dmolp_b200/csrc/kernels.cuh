// Host-side launchers of the DMOLP kernels (one translation unit per kernel family).
#pragma once

#include <utility>
#include <vector>

#include "device_state.cuh"

namespace dmolp {

// ---- host (hubsort.cpp) ----
// find_hub_nodes on (vertex, degree) pairs in the reference's map order, std::sort's tie order kept.
std::vector<int> hubs_from_pairs(std::vector<std::pair<int, int>> sd);
// The same on the raw degrees of one rank (pairs in map order, vertex V-1 down to 0, built on all threads).
std::vector<int> hubs_from_degrees(const int32_t *degree, int64_t nv);
// The number of hubs of n vertices with the given sum and maximum of degrees; the sort's depth limit; and the rest of
// the top of its order from where the device left it (hubsort.cpp).
int64_t hub_count(int64_t n, int64_t total, int32_t dmax);
int introsort_depth(int64_t n);
void finish_top(std::pair<int32_t, int32_t> *a, int64_t m, int64_t t0, int64_t depth, int64_t cut, bool whole);
// find_first_seed's (vertex, degree) over that order, its id-vs-degree tie test included.
std::pair<int, int> first_seed_of(const int32_t *degree, int64_t nv);

// ---- window selection (select_kernels.cu) ----
// Records i < cnt->npos carry a segment bown[i] in [0,nseg) (or -1: an empty slot, ignored) and a 64-bit key
// bkey[i] whose top bit is below `keybits`; keys are unique.  `stopped` (may be null) turns the launch into a no-op
// once it is non-zero.
// The LP window straight out of the selection: the key of a selected record slot holds its vertex and
// degree (key = (dk << ibits) | v, dk = maxdeg - deg when RE[label] > 1, else deg; label = its segment);
// v is stamped sstamp[v] = t, appended to win / nwin and to its decision-class list dec[c] / ndec[c], and
// its degree added to *te.  The segments' needs are min(n, ceil(*ratio * n)) for n = npart[seg] (the
// reference's ceil(e^(-t/5) n), gpu_lp_boundary.cu:244).
struct SplitArgs {
    const double *RE;
    const int32_t *npart;
    const double *ratio;
    int32_t *sstamp;
    int32_t *win;
    int *nwin;
    int32_t *dec[3];
    int *ndec;
    unsigned long long *te;
    unsigned long long *wsum;  // += window_mix(v) for every selected v
    int t, eff, ibits, maxdeg;
};
// first_hist_ready: the writer of the records has already added every record's first digit (bits
// [select_first_shift(keybits), +8) of its key) into histogram buffer 0 of c->b.hist, bin seg * 256 + digit.
void select_window(dmolp_ctx *c, int nseg, int keybits, const SplitArgs &split, const int *stopped,
                   bool first_hist_ready);
inline int select_first_shift(int keybits) { return ((keybits + kRadixBits - 1) / kRadixBits - 1) * kRadixBits; }
void select_prepare();  // kernel attributes; call once before any capture
// The LP window by degree bins (k_select_deg): the same window as select_window, for at most
// kDegSelMaxK labels, with the boundary test's superbin counts in b.dsup (BndArgs::dsup).  Returns false
// (nothing launched) for more labels.
bool select_window_deg(dmolp_ctx *c, int nseg, const SplitArgs &split, const int *stopped);
int select_binary_version();  // sm version of the loaded device code (major * 10 + minor), -1 on failure

// ---- LP loop (lp_kernels.cu) ----
struct LpLaunch {
    int k;
    int eff;       // labels scored: min(k,32) or k
    int mode;      // DMOLP_LP_MODE_*
};
void lp_check_symmetric(dmolp_ctx *c, unsigned long long *counts);  // *b.flag: a reverse is missing
void lp_symmetry_hash(dmolp_ctx *c, unsigned long long *sum, unsigned long long key);  // *sum += the multiset sum
void lp_fill(dmolp_ctx *c, int32_t *p, int64_t n, int32_t v);
void lp_degrees(dmolp_ctx *c, const int64_t *off, int64_t nv, int32_t *deg);  // deg[v] = off[v+1] - off[v]
void lp_reset_stats(dmolp_ctx *c, int k, const int *stopped);
// use_hot: the hot labels are current (lp_hot_refresh since the labels were last set outside the loop)
// keep_eff > 0: also write the kept label counts vcnt (labels < keep_eff <= 32) of every non-hub vertex
void lp_stats(dmolp_ctx *c, int k, const int *stopped, const int *skip, bool use_hot = false, int keep_eff = 0,
              int hub_eff = 0);  // hub_eff > 0: also every hub's label counts (hh), labels < hub_eff
void lp_hot_hist(dmolp_ctx *c);              // b.degh = histogram of min(degree, 65535), degree > 0
void lp_hot_build(dmolp_ctx *c, int dstar);  // vertices of degree >= dstar ranked; colh; b.flag = their number
void lp_hot_refresh(dmolp_ctx *c);           // hot labels from the resident labels
void lp_init_end(dmolp_ctx *c, int mode);
void lp_hub_index(dmolp_ctx *c);            // b.hidx from bucket[2] (once per graph)
// keeps it current; otherwise the selected hubs' rows are recounted.
void lp_iteration(dmolp_ctx *c, const LpLaunch &L, int t, bool first, bool last);
// one-off pieces used by dmolp_window_select / dmolp_lp_apply
void lp_window_from_list(dmolp_ctx *c, int k, int t, const double *RE_dev, int nprev);
void lp_apply_list(dmolp_ctx *c, int k, int eff, int n);

// ---- LP loop in one launch (lp_loop.cu) ----
void loop_order(dmolp_ctx *c);  // slot orders (once per graph)
void loop_run(dmolp_ctx *c, const LpLaunch &L, int iters);  // every iteration, after the run-start statistics pass
void loop_prepare();  // kernel attributes

// ---- phase 1 (seed_kernels.cu) ----
// Sum and maximum of the raw degrees, and what find_first_seed's closed form needs, to *b.hubst.
void p1_hub_stats(dmolp_ctx *c);
// The first steps of the hub sort on pairs (vertex, degree) in the reference's order, built in b.dlkey: Hoare
// partitions as long as the right side holds position t0 and more than kHubHostMax pairs are left; the state to
// *b.hubst.
void p1_hub_top(dmolp_ctx *c, int64_t t0, int depth);
// Seeds by the reference rule from b.hubs[0, nhubs) and the first seed: b.need[0, found), found = p1cnt[6].
// b.covered, b.best, p1cnt and, unless the rows are strictly increasing, b.claim are cleared by the caller.
void p1_find_seeds(dmolp_ctx *c, int k, int first, int64_t nhubs);
// Every growth round from the seeds b.need[0, k): labels, part sizes, the number of rounds in p1cnt[5].
void p1_grow(dmolp_ctx *c, int k, int theta);
void p1_prepare();  // kernel attributes

}  // namespace dmolp
