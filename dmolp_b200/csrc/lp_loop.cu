// Phase-2 label propagation with all iterations in one cooperative launch, for symmetric graphs of up to
// kLoopMaxArcs arcs.
//
// What bounds such a graph is not memory: an iteration's arcs and vertices are in L2, and the launch-per-step form
// (lp_kernels.cu) spends its 57 us an iteration (55 K-vertex mesh, 8 parts) on seven kernels' fill, drain and fixed
// work.  Here an iteration is three steps between grid barriers, four when more than 32 labels are scored:
//
//   turn    (no barrier of its own) every block ends the previous iteration and computes the penalties by itself
//   scan    every record slot: candidacy, the boundary test, the label's record count of this block
//   select  per label the need_p smallest (degree, id) records join the window: the slots are in that order, so a
//           record is taken when fewer than need_p records of its label precede it -- in the blocks before (the
//           counts of the scan), in the warps before, in its warp.  Decided on the spot from kept label counts when
//           at most 32 labels are scored
//   decide  (more than 32 labels) the window's rows are counted: a lane per row of at most 32 arcs, a warp per
//           longer one, hubs from their kept counts
//   update  the movers' arcs (cut, part counts, the neighbours' counts) and, in the same step, the next iteration's
//           candidate stamps from the window's rows: kGroup lanes per row of at most kLoopShort arcs, a warp per
//           queued piece of kLoopPiece arcs of a longer one
//
// The slot orders (ascending degree, descending degree; ids ascending among equals) are made once per graph by a
// stable radix sort of the vertices with arcs (k_loop_order).  A mover's new label is kept as (iteration, label) in
// pend[]: it counts from the next scan on, whose ascending walk also writes it to label[]; so no step rewrites what
// another thread of the same step reads.  Results are those of the launch-per-step form, bit for bit.
//
// Measured on B200, whole phase-2 calls: figures at use_loop (dmolp_cabi.cu), where the choice is made.
#include <algorithm>
#include <cfloat>

#include "select_radix.cuh"

namespace dmolp {
namespace {

constexpr int kLoopThreads = 512;
constexpr int kLoopWarps = kLoopThreads / 32;
constexpr int kOrderThreads = 1024;
constexpr int kOrderWarps = kOrderThreads / 32;
constexpr int kLoopBlockV = 256;  // record slots per block of a small graph
constexpr int kGroup = 4;         // lanes per row of the update
constexpr int kLaneRow = 32;      // decide: rows of at most this many arcs take one lane

// The slice [lo, hi) of n items that part i of m owns, in multiples of `unit`.
__device__ __forceinline__ void slice_of(int n, int i, int m, int unit, int &lo, int &hi) {
    const int len = ((n + m - 1) / m + unit - 1) / unit * unit;
    lo = min(n, i * len);
    hi = min(n, lo + len);
}

// ------------------------------------------------------------------------------------ slot order
struct OrderArgs {
    const int64_t *off;
    const int32_t *ball;     // vertices with arcs, ids ascending among equal degrees
    int2 *buf[2];            // [npos] (vertex, degree), scratch
    int32_t *first, *last;   // [max degree + 1] of each degree, scratch
    int2 *asc, *desc;        // [npos] out
    int *blk;                // [256 * grid] digit counts of every block, scratch
    int npos, npass;
    LpControl *ctl;
    unsigned int polls;
};

// Stable LSD radix sort by degree, 8 bits a pass: per pass the blocks' digit counts, a grid barrier, every block's
// own prefix over them, the scatter, a grid barrier.  Then the descending order: the groups of equal degree reversed.
__global__ void __launch_bounds__(kOrderThreads, 1) k_loop_order(OrderArgs a) {
    __shared__ int s_cnt[kOrderWarps][256];
    __shared__ int s_tot[256], s_base[256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x, n = a.npos;
    const unsigned below = (1u << lane) - 1;
    int lo, hi, wlo, whi;
    slice_of(n, blockIdx.x, G, 1, lo, hi);
    slice_of(hi - lo, w, kOrderWarps, 32, wlo, whi);
    wlo += lo;
    whi += lo;
    for (int q = 0; q < a.npass; ++q) {
        const int2 *const src = a.buf[q & 1];
        int2 *const dst = q + 1 < a.npass ? a.buf[(q + 1) & 1] : a.asc;
        auto load = [&](int i) {
            if (q) return src[i];
            const int v = a.ball[i];
            return make_int2(v, (int)(a.off[v + 1] - a.off[v]));
        };
        for (int d = lane; d < 256; d += 32) s_cnt[w][d] = 0;
        __syncwarp();
        for (int i0 = wlo; i0 < whi; i0 += 32) {
            const int i = i0 + lane;
            const int d = i < whi ? (load(i).y >> (8 * q)) & 255 : -1;
            const unsigned m = __match_any_sync(DMOLP_FULL_MASK, d);
            if (d >= 0 && lane == __ffs(m) - 1) s_cnt[w][d] += __popc(m);
            __syncwarp();
        }
        __syncthreads();
        for (int d = threadIdx.x; d < 256; d += blockDim.x) {
            int run = 0;
            for (int j = 0; j < kOrderWarps; ++j) {
                const int c = s_cnt[j][d];
                s_cnt[j][d] = run;
                run += c;
            }
            a.blk[d * G + blockIdx.x] = run;
        }
        if (!grid_sync(a.ctl, a.polls, 40)) return;
        for (int d = w; d < 256; d += kOrderWarps) {
            int tot = 0, before = 0;
            for (int j = lane; j < G; j += 32) {
                const int c = __ldcg(a.blk + d * G + j);
                tot += c;
                before += j < (int)blockIdx.x ? c : 0;
            }
            for (int o = 16; o > 0; o >>= 1) {
                tot += __shfl_xor_sync(DMOLP_FULL_MASK, tot, o);
                before += __shfl_xor_sync(DMOLP_FULL_MASK, before, o);
            }
            if (lane == 0) {
                s_tot[d] = tot;
                s_base[d] = before;
            }
        }
        __syncthreads();
        if (w == 0) {  // exclusive prefix of the 256 totals, 8 per lane
            int c[8], sum = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                c[j] = s_tot[lane * 8 + j];
                sum += c[j];
            }
            int incl = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
                if (lane >= o) incl += y;
            }
            int run = incl - sum;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                s_base[lane * 8 + j] += run;
                run += c[j];
            }
        }
        __syncthreads();
        for (int i0 = wlo; i0 < whi; i0 += 32) {
            const int i = i0 + lane;
            int2 x = make_int2(0, 0);
            int d = -1;
            if (i < whi) {
                x = load(i);
                d = (x.y >> (8 * q)) & 255;
            }
            const unsigned m = __match_any_sync(DMOLP_FULL_MASK, d);
            const int r = d >= 0 ? s_base[d] + s_cnt[w][d] + __popc(m & below) : 0;
            __syncwarp();
            if (d >= 0 && lane == __ffs(m) - 1) s_cnt[w][d] += __popc(m);
            __syncwarp();
            if (d >= 0) dst[r] = x;
        }
        if (!grid_sync(a.ctl, a.polls, 41)) return;
    }
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = G * blockDim.x;
    for (int i = t0; i < n; i += nt) {
        const int d = a.asc[i].y;
        if (i == 0 || a.asc[i - 1].y != d) a.first[d] = i;
        if (i == n - 1 || a.asc[i + 1].y != d) a.last[d] = i;
    }
    if (!grid_sync(a.ctl, a.polls, 42)) return;
    for (int i = t0; i < n; i += nt) {
        const int2 x = a.asc[i];
        a.desc[(n - 1 - a.last[x.y]) + (i - a.first[x.y])] = x;
    }
}

// ------------------------------------------------------------------------------------ the loop
// The counters of one iteration (by parity).
struct LoopCnt {
    int nwin, nmov, nwp, nmp, nbig;  // window, movers, their queued row pieces, window rows of more than kLaneRow arcs
    int ncand, nbnd;
    unsigned long long te_cand, te_sel, wsum, arcs_dec, arcs_upd;
};

struct LoopArgs {
    const int2 *ord[2];      // (vertex, degree): ascending, descending
    int16_t *lab[2];         // [npos] label of a slot's record of this order's direction, -1: none
    int *blk;                // [k * grid] records per label and block
    uint32_t *pend;          // [nv] iteration << 10 | new label
    int32_t *win, *big, *mov;
    int2 *wpiece, *mpiece;   // (vertex, first arc)
    LoopCnt *cnt;            // [2]
    long long narcs;
    int npos, nv, k, eff, mode, iters, kept, hubs;
    unsigned int polls;
};

// Shared memory of k_lp_loop: the per-label arrays, then the warps' label counters [kLoopWarps][k].
__host__ __device__ constexpr size_t loop_smem(int k) {
    return (size_t)k * (2 * sizeof(double) + 2 * sizeof(long long) + 2 * sizeof(int)) +
           (size_t)kLoopWarps * k * sizeof(int);
}

// Slots for cnt entries per lane from a global counter, one atomic per warp (all lanes call it).
__device__ __forceinline__ int warp_reserve(int *ctr, int cnt) {
    const int lane = threadIdx.x & 31;
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
        if (lane >= o) incl += y;
    }
    int base = 0;
    if (lane == 31 && incl) base = atomicAdd(ctr, incl);
    return __shfl_sync(DMOLP_FULL_MASK, base, 31) + incl - cnt;
}

__device__ __forceinline__ int warp_reserve1(int *ctr, bool pred) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(DMOLP_FULL_MASK, pred);
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(ctr, __popc(m));
    return __shfl_sync(DMOLP_FULL_MASK, base, 0) + __popc(m & ((1u << lane) - 1));
}

__device__ __forceinline__ void queue_pieces(int2 *q, int at, int v, int deg) {
    for (int j = 0; j < deg; j += kLoopPiece) q[at++] = make_int2(v, j);
}

__device__ __forceinline__ int pieces_of(int deg) { return deg > kLoopShort ? (deg + kLoopPiece - 1) / kLoopPiece : 0; }

// The rule of warp_argmax over labels < eff in one thread, from counts cnt(c); own: the vertex's label.  Returns the
// new label, or own.
template <typename C>
__device__ __forceinline__ int decide_counts(int eff, const double *tp, int own, C cnt) {
    double best = -DBL_MAX;
    int bkey = 0x7fffffff, blab = -1, own_cnt = 0;
    for (int c = 0; c < eff; ++c) {
        const int n = cnt(c);
        if (c == own) own_cnt = n;
        const double sc = n > 0 ? __dmul_rn((double)n, tp[c]) : 0.0;
        const int key = tiekey(c);
        if (better(sc, key, best, bkey)) {
            best = sc;
            bkey = key;
            blab = c;
        }
    }
    const double own_raw = (unsigned)own < (unsigned)eff ? (double)own_cnt : -1e300;
    return best > own_raw ? blab : own;
}

// The same from 32 kept 16-bit counts: labels with neighbours, and the others only against an own label that is not
// scored (a scored own label's count is never below their score of 0).
__device__ __forceinline__ int decide_kept(int eff, const double *tp, int own, const uint4 (&c4)[4]) {
    double best = -DBL_MAX;
    int bkey = 0x7fffffff, blab = -1, own_cnt = 0;
#pragma unroll
    for (int c = 0; c < 32; ++c) {
        const uint4 y = c4[c >> 3];
        const uint32_t word = (c & 6) == 0 ? y.x : (c & 6) == 2 ? y.y : (c & 6) == 4 ? y.z : y.w;
        const int n = (int)((word >> (16 * (c & 1))) & 0xffffu);
        if (c == own) own_cnt = n;
        if (c < eff && (n > 0 || own >= eff)) {
            const double sc = n > 0 ? __dmul_rn((double)n, tp[c]) : 0.0;
            if (better(sc, tiekey(c), best, bkey)) {
                best = sc;
                bkey = tiekey(c);
                blab = c;
            }
        }
    }
    return blab >= 0 && best > (own < eff ? (double)own_cnt : -1e300) ? blab : own;
}

// The same from the neighbours' labels l[0, R) (-1: none) of a row: only labels seen can win over a scored own label.
template <int R>
__device__ __forceinline__ int decide_row(const double *tp, int own, const int (&l)[R], int deg) {
    double best = -DBL_MAX;
    int bkey = 0x7fffffff, blab = -1, own_cnt = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) own_cnt += l[j] == own;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        if (j >= deg) break;
        const int c = l[j];
        int n = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) n += l[i] == c;
        const double sc = __dmul_rn((double)n, tp[c]);
        const int key = tiekey(c);
        if (better(sc, key, best, bkey)) {
            best = sc;
            bkey = key;
            blab = c;
        }
    }
    return blab >= 0 && best > (double)own_cnt ? blab : own;
}

__global__ void __launch_bounds__(kLoopThreads, 1) k_lp_loop(Buffers b, LoopArgs a) {
    extern __shared__ double s_dyn[];
    const int k = a.k, eff = a.eff, G = gridDim.x, B = blockIdx.x;
    double *const s_re = s_dyn, *const s_tp = s_re + k;
    long long *const s_vc = reinterpret_cast<long long *>(s_tp + k), *const s_in = s_vc + k;  // this block's changes
    int *const s_need = reinterpret_cast<int *>(s_in + k), *const s_base = s_need + k, *const s_w = s_base + k;
    __shared__ int s_stop;
    __shared__ unsigned long long s_sum[kLoopWarps][4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gwarp = w * G + B, nwarp = kLoopWarps * G;  // the blocks' first warps first: short lists spread
    const unsigned below = (1u << lane) - 1;
    int *const s_my = s_w + w * k;
    LpControl *const ctl = b.ctrl;
    // The slot orders' launch of the same call gave up at one of its barriers: the orders hold no ids of this graph.
    if (*(volatile int *)&ctl->wait_timeout) return;

    // ---- start (the statistics pass has run) ----
    long long prev_cut = 0;
    int conv = 0, reason = 0, iters = 0;  // thread 0 of every block, alike
    const int bad0 = (b.cnt->cut_arcs & 1ull) || ctl->error;
    for (int v = B * kLoopThreads + threadIdx.x; v < a.nv; v += G * kLoopThreads) {
        b.stamp[v] = 0;   // read from the second iteration on
        a.pend[v] = 0u;
    }
    for (int p = threadIdx.x; p < k; p += kLoopThreads) s_vc[p] = s_in[p] = 0;
    prev_cut = (long long)(b.cnt->cut_arcs >> 1);
    int lo, hi, wlo, whi;
    slice_of(a.npos, B, G, 1, lo, hi);
    slice_of(hi - lo, w, kLoopWarps, 32, wlo, whi);
    wlo += lo;
    whi += lo;
    // warp sums of four values added to the iteration's counters, one atomic per block and value
    auto block_sums = [&](unsigned long long x0, unsigned long long x1, unsigned long long x2, unsigned long long x3,
                          auto add) {
        x0 = warp_sum_u64(x0);
        x1 = warp_sum_u64(x1);
        x2 = warp_sum_u64(x2);
        x3 = warp_sum_u64(x3);
        if (lane == 0) {
            s_sum[w][0] = x0;
            s_sum[w][1] = x1;
            s_sum[w][2] = x2;
            s_sum[w][3] = x3;
        }
        __syncthreads();
        if (threadIdx.x < 4) {
            unsigned long long s = 0;
            for (int j = 0; j < kLoopWarps; ++j) s += s_sum[j][threadIdx.x];
            if (s) add((int)threadIdx.x, s);
        }
    };

    int t = 1;
    for (;; ++t) {
        LoopCnt *const cn = &a.cnt[t & 1], *const pc = &a.cnt[(t + 1) & 1];  // this iteration's, the previous one's
        // ---- turn: end of iteration t - 1 (phase2.cpp:309-415) by thread 0, penalties of t by warp 1 meanwhile ----
        if (w == 1 && t <= a.iters && !bad0)
            warp_penalties(k, [&](int p) { return sll(__ldcg(b.vc + p)); },
                           [&](int p) { return sll(__ldcg(b.intra + p)) / 2; }, b.logtab[t], s_re, s_tp,
                           B == 0 ? b.penhist + (size_t)(t - 1) * DMOLP_MAX_K : nullptr);
        for (int p = lane; p < k; p += 32) s_my[p] = 0;
        if (threadIdx.x == 0) {
            int stop = bad0 ? 4 : 0;
            if (t > 1 && !stop) {
                const int win = __ldcg(&pc->nwin), mov = __ldcg(&pc->nmov);
                const unsigned long long arcs = __ldcg(&b.cnt->cut_arcs);
                bool stats = true;
                if (win == 0) {
                    stats = false;
                    if (a.mode == DMOLP_LP_MODE_REF) stop = 1;
                } else if (mov == 0 && a.mode == DMOLP_LP_MODE_REF) {
                    stats = false;
                    stop = 2;
                }
                if (stats) {
                    if (arcs & 1ull) {
                        stop = 4;
                    } else {
                        const long long cur = (long long)(arcs >> 1);
                        const double delta =
                            prev_cut > 0 ? fabs(__ddiv_rn((double)(cur - prev_cut), (double)prev_cut)) : 1.0;
                        conv = delta < 0.03 ? conv + 1 : 0;
                        prev_cut = cur;
                        if (a.mode == DMOLP_LP_MODE_REF && conv >= 10) stop = 3;
                    }
                }
                iters = t - 1;
                if (B == 0) {
                    LpRecordDev &r = b.rec[t - 2];
                    r.iteration = t - 1;
                    r.window = win;
                    r.candidates = t == 2 ? -1 : __ldcg(&pc->ncand);
                    r.changes = mov;
                    r.boundary = __ldcg(&pc->nbnd);
                    r.edge_cut = prev_cut;
                    const unsigned long long sel = __ldcg(&pc->te_sel);
                    r.te_prev = t == 2 ? (unsigned long long)a.narcs : b.rec[t - 3].te_sel;
                    r.te_cand = __ldcg(&pc->te_cand);
                    r.te_sel = sel;
                    r.te_stats = stats ? (unsigned long long)a.narcs : 0;
                    r.arcs_bnd = 0;
                    r.arcs_dec = __ldcg(&pc->arcs_dec);
                    r.arcs_upd = __ldcg(&pc->arcs_upd);
                    r.arcs_mark = t == 2 ? 0 : r.te_prev;  // every window row was walked
                    r.te_hubsel = 0;
                    r.win_sum = __ldcg(&pc->wsum);
                    if (stop == 4) ctl->error = 1;
                }
            }
            reason = stop;
            s_stop = stop || t > a.iters;
        }
        __syncthreads();
        if (B == 0 && t > 1 && !bad0) {
            long long *const ch = b.cnthist + (size_t)(t - 2) * 2 * DMOLP_MAX_K;
            for (int p = threadIdx.x; p < k; p += kLoopThreads) {
                ch[p] = sll(__ldcg(b.vc + p));
                ch[DMOLP_MAX_K + p] = sll(__ldcg(b.intra + p)) / 2;
            }
        }
        if (s_stop) break;  // the same in every block
        bool has_desc = false;
        for (int p = threadIdx.x; p < k; p += kLoopThreads) has_desc |= s_re[p] > 1.0;
        has_desc = __syncthreads_or(has_desc);

        // ---- scan: candidates (t = 1: all; else stamped) with a neighbour of another label
        //      (gpu_lp_boundary.cu:195-270), counted per label in their label's order ----
        {
            unsigned long long te = 0, nc = 0, nb = 0;
            auto count = [&](int lab) {
                const unsigned m = __match_any_sync(DMOLP_FULL_MASK, lab);
                if (lab >= 0 && lane == __ffs(m) - 1) s_my[lab] += __popc(m);
                __syncwarp();
            };
            auto own_of = [&](int lv, uint32_t pe) {
                return t > 1 && (int)(pe >> 10) == t - 1 ? (int)(pe & 1023u) : lv;
            };
            // per step 32 slots of either order (the descending one only when a label takes its largest degrees)
            for (int i0 = wlo; i0 < whi; i0 += 32) {
                const int i = i0 + lane;
                const bool in = i < whi;
                int2 x[2];
                int st[2], nd[2], lv[2];
                uint32_t pe[2];
                x[0] = in ? a.ord[0][i] : make_int2(0, 0);
                x[1] = in && has_desc ? a.ord[1][i] : make_int2(0, 0);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    st[q] = b.stamp[x[q].x];
                    nd[q] = b.ndiff[x[q].x];
                    lv[q] = b.label[x[q].x];  // (of a mover of the last iteration: not used, see pend)
                    pe[q] = a.pend[x[q].x];
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q == 1 && !has_desc) break;
                    const int own = own_of(lv[q], pe[q]);
                    const bool cand = in && (t == 1 || st[q] == t), isb = cand && nd[q] > 0;
                    if (q == 0) {
                        if (in && own != lv[0]) b.label[x[0].x] = own;  // the last iteration's movers
                        nc += cand;
                        nb += isb;
                        te += cand ? (unsigned long long)x[0].y : 0;
                    }
                    const int lab = isb && (s_re[own] > 1.0) == (q == 1) ? own : -1;
                    if (in) a.lab[q][i] = (int16_t)lab;
                    count(lab);
                }
            }
            block_sums(nc, nb, te, 0, [&](int j, unsigned long long s) {
                if (j == 0) atomicAdd(&cn->ncand, (int)s);
                else if (j == 1) atomicAdd(&cn->nbnd, (int)s);
                else atomicAdd(&cn->te_cand, s);
            });
            // (a barrier in block_sums: every warp has counted) this block's counts, the warps' starts in it
            for (int p = threadIdx.x; p < k; p += kLoopThreads) {
                int run = 0;
                for (int j = 0; j < kLoopWarps; ++j) {
                    const int c = s_w[j * k + p];
                    s_w[j * k + p] = run;
                    run += c;
                }
                a.blk[p * G + B] = run;
            }
        }
        if (!grid_sync(ctl, a.polls, 43)) return;
        // the previous iteration's counters were read before the barrier
        if (B == 0 && threadIdx.x == 0) *pc = LoopCnt();

        // ---- select: need[p] = min(n_p, ceil(e^(-t/5) n_p)) records (gpu_lp_boundary.cu:244, 277-301) ----
        for (int p = w; p < k; p += kLoopWarps) {
            int tot = 0, before = 0;
            for (int j = lane; j < G; j += 32) {
                const int c = __ldcg(a.blk + p * G + j);
                tot += c;
                before += j < B ? c : 0;
            }
            for (int o = 16; o > 0; o >>= 1) {
                tot += __shfl_xor_sync(DMOLP_FULL_MASK, tot, o);
                before += __shfl_xor_sync(DMOLP_FULL_MASK, before, o);
            }
            if (lane == 0) {
                const int m = (int)ceil(__dmul_rn(b.ratiotab[t], (double)tot));
                s_need[p] = m > tot ? tot : m;
                s_base[p] = before;
            }
        }
        __syncthreads();
        {
            unsigned long long te = 0, ws = 0;
            // 32 slots of either order a step, as in the scan
            for (int i0 = wlo; i0 < whi; i0 += 32) {
                const int i = i0 + lane;
                int lab[2], nl[2];
                lab[0] = i < whi ? (int)a.lab[0][i] : -1;
                lab[1] = i < whi && has_desc ? (int)a.lab[1][i] : -1;
                if (!__any_sync(DMOLP_FULL_MASK, lab[0] >= 0 || lab[1] >= 0)) continue;
                bool take[2];
                unsigned mt[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const unsigned m = __match_any_sync(DMOLP_FULL_MASK, lab[q]);
                    take[q] = lab[q] >= 0 && s_base[lab[q]] + s_my[lab[q]] + __popc(m & below) < s_need[lab[q]];
                    __syncwarp();
                    if (lab[q] >= 0 && lane == __ffs(m) - 1) s_my[lab[q]] += __popc(m);
                    __syncwarp();
                    mt[q] = __ballot_sync(DMOLP_FULL_MASK, take[q]);
                    nl[q] = lab[q];
                }
                if (!(mt[0] | mt[1])) continue;
                int wbase = 0;  // needed only at the end of the step
                if (lane == 0) wbase = atomicAdd(&cn->nwin, __popc(mt[0]) + __popc(mt[1]));
                int2 x[2];
                int np[2], hub[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) x[q] = take[q] ? a.ord[q][i] : make_int2(0, 0);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    hub[q] = take[q] && a.kept && a.hubs ? b.hidx[x[q].x] : -1;
                    np[q] = take[q] ? pieces_of(x[q].y) : 0;
                    if (take[q]) {
                        te += (unsigned long long)x[q].y;
                        ws += window_mix(x[q].x);
                    }
                }
                if (a.kept) {
                    uint4 c4[2][4];
#pragma unroll
                    for (int q = 0; q < 2; ++q)
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            c4[q][r] = make_uint4(0, 0, 0, 0);
                            if (take[q] && r * 8 < eff)
                                c4[q][r] = reinterpret_cast<const uint4 *>(b.vcnt + (size_t)x[q].x * 32)[r];
                        }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        if (!take[q]) continue;
                        if (hub[q] >= 0) {
                            const int32_t *const row = b.hh + (size_t)hub[q] * DMOLP_MAX_K;
                            nl[q] = decide_counts(eff, s_tp, lab[q], [&](int c) { return row[c]; });
                        } else {
                            nl[q] = decide_kept(eff, s_tp, lab[q], c4[q]);
                        }
                    }
                }
                const bool mv[2] = {nl[0] != lab[0], nl[1] != lab[1]};
                const unsigned mm[2] = {__ballot_sync(DMOLP_FULL_MASK, mv[0]), __ballot_sync(DMOLP_FULL_MASK, mv[1])};
                const bool big[2] = {!a.kept && take[0] && x[0].y > kLaneRow, !a.kept && take[1] && x[1].y > kLaneRow};
                const unsigned mb[2] = {__ballot_sync(DMOLP_FULL_MASK, big[0]), __ballot_sync(DMOLP_FULL_MASK, big[1])};
                // movers (kept counts) or long rows (else): one list of the two is filled
                int lbase = 0;
                if (lane == 0 && (mm[0] | mm[1])) lbase = atomicAdd(&cn->nmov, __popc(mm[0]) + __popc(mm[1]));
                if (lane == 0 && (mb[0] | mb[1])) lbase = atomicAdd(&cn->nbig, __popc(mb[0]) + __popc(mb[1]));
                wbase = __shfl_sync(DMOLP_FULL_MASK, wbase, 0);
                lbase = __shfl_sync(DMOLP_FULL_MASK, lbase, 0);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (take[q]) a.win[wbase + __popc(mt[q] & below)] = x[q].x;
                    if (big[q]) a.big[lbase + __popc(mb[q] & below)] = x[q].x;
                    if (mv[q]) {
                        a.mov[lbase + __popc(mm[q] & below)] = x[q].x;
                        a.pend[x[q].x] = (uint32_t)t << 10 | (uint32_t)nl[q];
                        atomicAdd((unsigned long long *)&s_vc[lab[q]], ~0ull);
                        atomicAdd((unsigned long long *)&s_vc[nl[q]], 1ull);
                    }
                    wbase += __popc(mt[q]);
                    lbase += __popc(mm[q]) + __popc(mb[q]);
                }
                if (__any_sync(DMOLP_FULL_MASK, np[0] + np[1] > 0)) {
                    const int at = warp_reserve(&cn->nwp, np[0] + np[1]);
                    if (np[0]) queue_pieces(a.wpiece, at, x[0].x, x[0].y);
                    if (np[1]) queue_pieces(a.wpiece, at + np[0], x[1].x, x[1].y);
                    const int p0 = mv[0] ? np[0] : 0, p1 = mv[1] ? np[1] : 0;
                    const int am = warp_reserve(&cn->nmp, p0 + p1);
                    if (p0) queue_pieces(a.mpiece, am, x[0].x, x[0].y);
                    if (p1) queue_pieces(a.mpiece, am + p0, x[1].x, x[1].y);
                }
            }
            block_sums(te, ws, 0, 0, [&](int j, unsigned long long s) { atomicAdd(j == 0 ? &cn->te_sel : &cn->wsum, s); });
        }
        if (!grid_sync(ctl, a.polls, 44)) return;
        const int nwin = __ldcg(&cn->nwin);

        if (!a.kept) {
            // ---- decide (every label scored): boundaryLPKernel_unified's rule (gpu_lp_boundary.cu:354-426) ----
            unsigned long long rd = 0;
            auto move_to = [&](bool mv, int v, int own, int nl, int deg) {  // all lanes
                if (!__any_sync(DMOLP_FULL_MASK, mv)) return;
                const int slot = warp_reserve1(&cn->nmov, mv);
                const int np = mv ? pieces_of(deg) : 0;
                const int q = warp_reserve(&cn->nmp, np);
                if (mv) {
                    a.mov[slot] = v;
                    a.pend[v] = (uint32_t)t << 10 | (uint32_t)nl;
                    if (np) queue_pieces(a.mpiece, q, v, deg);
                    atomicAdd((unsigned long long *)&s_vc[own], ~0ull);
                    atomicAdd((unsigned long long *)&s_vc[nl], 1ull);
                }
            };
            const int nbig = __ldcg(&cn->nbig);
            // one warp takes a long row or 32 short ones
            const int nitem = nbig + (nwin + 31) / 32;
            for (int it = gwarp; it < nitem; it += nwarp) {
                if (it < nbig) {
                    const int v = a.big[it], own = b.label[v];
                    const int64_t s = b.off[v], e = b.off[v + 1];
                    const int hi_ = a.hubs ? b.hidx[v] : -1;
                    double best;
                    int blab, own_cnt;
                    if (hi_ >= 0) {
                        const int32_t *const row = b.hh + (size_t)hi_ * DMOLP_MAX_K;
                        warp_argmax(eff, s_tp, lane, [&](int c) { return row[c]; }, best, blab);
                        own_cnt = row[own];
                    } else {
                        for (int c = lane; c < k; c += 32) s_my[c] = 0;
                        __syncwarp();
                        for (int64_t j0 = s + lane; j0 < e; j0 += 256) {
                            int u[8], l[8];
    #pragma unroll
                            for (int q = 0; q < 8; ++q) u[q] = j0 + q * 32 < e ? __ldg(b.col + j0 + q * 32) : -1;
    #pragma unroll
                            for (int q = 0; q < 8; ++q) l[q] = u[q] >= 0 ? b.label[u[q]] : -1;
    #pragma unroll
                            for (int q = 0; q < 8; ++q)
                                if (l[q] >= 0) atomicAdd(&s_my[l[q]], 1);
                        }
                        __syncwarp();
                        warp_argmax(eff, s_tp, lane, [&](int c) { return s_my[c]; }, best, blab);
                        own_cnt = s_my[own];
                        if (lane == 0) rd += (unsigned long long)(e - s);
                        __syncwarp();
                    }
                    move_to(lane == 0 && best > (double)own_cnt && blab != own, v, own, blab, (int)(e - s));
                    continue;
                }
                const int i = (it - nbig) * 32 + lane;
                int v = 0, own = 0, deg = 0, nl = 0;
                if (i < nwin) {
                    v = a.win[i];
                    own = nl = b.label[v];
                    const int64_t s = b.off[v];
                    deg = (int)(b.off[v + 1] - s);
                    if (deg <= kLaneRow) {
                        rd += (unsigned long long)deg;
                        int l[kLaneRow];
#pragma unroll
                        for (int j = 0; j < 16; ++j) l[j] = j < deg ? __ldg(b.col + s + j) : -1;
#pragma unroll
                        for (int j = 0; j < 16; ++j) l[j] = l[j] >= 0 ? b.label[l[j]] : -1;
                        if (deg <= 16) {
                            int h[16];
#pragma unroll
                            for (int j = 0; j < 16; ++j) h[j] = l[j];
                            nl = decide_row<16>(s_tp, own, h, deg);
                        } else {
#pragma unroll
                            for (int j = 16; j < kLaneRow; ++j) l[j] = j < deg ? __ldg(b.col + s + j) : -1;
#pragma unroll
                            for (int j = 16; j < kLaneRow; ++j) l[j] = l[j] >= 0 ? b.label[l[j]] : -1;
                            nl = decide_row<kLaneRow>(s_tp, own, l, deg);
                        }
                    }
                }
                move_to(nl != own, v, own, nl, deg);
            }
            block_sums(rd, 0, 0, 0, [&](int, unsigned long long s) { atomicAdd(&cn->arcs_dec, s); });
            if (!grid_sync(ctl, a.polls, 45)) return;
        }

        // ---- update: the movers' arcs (see k_update in lp_kernels.cu: weight 2 when the neighbour stays, 1 when it
        //      moves too), kGroup lanes per row; then the stamps of iteration t + 1 ----
        {
            long long dcut = 0;
            unsigned long long rd = 0;
            // the arcs s + first, s + first + step, ... < e of a mover from label x to c; U in flight
            auto mover_arcs = [&](int x, int c, int64_t s, int64_t e, int first, int step, long long &in_c,
                                  long long &out_a, int &dv) {
                for (int64_t j0 = s + first; j0 < e; j0 += 4 * step) {
                    int u[4], lu[4], hu[4];
                    uint32_t pu[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) u[q] = j0 + q * step < e ? __ldg(b.col + j0 + q * step) : -1;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        lu[q] = u[q] >= 0 ? b.label[u[q]] : 0;
                        pu[q] = u[q] >= 0 ? a.pend[u[q]] : 0u;
                        hu[q] = u[q] >= 0 && a.hubs ? b.hidx[u[q]] : -1;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (u[q] < 0) continue;
                        const bool moves = (int)(pu[q] >> 10) == t;
                        const int ln = moves ? (int)(pu[q] & 1023u) : lu[q], wt = moves ? 1 : 2;
                        dcut += wt * ((int)(c != ln) - (int)(x != lu[q]));
                        in_c += wt * (int)(c == ln);
                        out_a += wt * (int)(x == lu[q]);
                        const int du = (int)(ln != c) - (int)(lu[q] != x);
                        if (du) atomicAdd(&b.ndiff[u[q]], du);
                        if (!moves) dv += (int)(c != lu[q]) - (int)(x != lu[q]);
                        if (hu[q] >= 0) {
                            int32_t *const row = b.hh + (size_t)hu[q] * DMOLP_MAX_K;
                            if (x < eff) atomicAdd(&row[x], -1);
                            if (c < eff) atomicAdd(&row[c], 1);
                        } else if (a.kept) {
                            uint32_t *const wd = reinterpret_cast<uint32_t *>(b.vcnt + (size_t)u[q] * 32);
                            const uint32_t da = x < eff ? 1u << ((x & 1) * 16) : 0u;
                            const uint32_t dc = c < eff ? 1u << ((c & 1) * 16) : 0u;
                            if (da && dc && (x >> 1) == (c >> 1)) {
                                atomicAdd(&wd[x >> 1], dc - da);
                            } else {
                                if (da) atomicSub(&wd[x >> 1], da);
                                if (dc) atomicAdd(&wd[c >> 1], dc);
                            }
                        }
                    }
                }
            };
            // sums over the lanes of a group, added by its first lane
            auto mover_done = [&](int width, int v, int x, int c, long long in_c, long long out_a, int dv) {
                for (int o = width >> 1; o > 0; o >>= 1) {
                    in_c += __shfl_xor_sync(DMOLP_FULL_MASK, in_c, o);
                    out_a += __shfl_xor_sync(DMOLP_FULL_MASK, out_a, o);
                    dv += __shfl_xor_sync(DMOLP_FULL_MASK, dv, o);
                }
                if ((lane & (width - 1)) == 0) {
                    if (dv) atomicAdd(&b.ndiff[v], dv);
                    if (in_c) atomicAdd((unsigned long long *)&s_in[c], (unsigned long long)in_c);
                    if (out_a) atomicAdd((unsigned long long *)&s_in[x], (unsigned long long)(-out_a));
                }
            };
            const int nmov = __ldcg(&cn->nmov), nmp = __ldcg(&cn->nmp), nwp = __ldcg(&cn->nwp);
            constexpr int kRows = 32 / kGroup;
            // little to do: half of the warps take the movers, half the window, so their chains of loads overlap
            const int half = nwarp / 2;
            const bool split = nmov + nmp * kRows <= half * kRows && nwin + nwp * kRows <= 2 * half * kRows;
            const int mw = split ? (gwarp < half ? gwarp : nmov + nmp) : gwarp, ms = split ? half : nwarp;
            const int ww = split ? (gwarp >= half ? gwarp - half : nwin + nwp) : gwarp;
            for (int q = mw; q < nmp; q += ms) {
                const int2 y = a.mpiece[q];
                const int64_t s = b.off[y.x] + y.y, e = min((long long)b.off[y.x + 1], (long long)s + kLoopPiece);
                const int x = b.label[y.x], c = (int)(a.pend[y.x] & 1023u);
                long long in_c = 0, out_a = 0;
                int dv = 0;
                mover_arcs(x, c, s, e, lane, 32, in_c, out_a, dv);
                mover_done(32, y.x, x, c, in_c, out_a, dv);
                if (lane == 0) rd += (unsigned long long)(e - s);
            }
            for (int i0 = mw * kRows; i0 < nmov; i0 += ms * kRows) {
                const int i = i0 + lane / kGroup;
                int v = 0, x = 0, c = 0;
                int64_t s = 0, e = 0;
                if (i < nmov) {
                    v = a.mov[i];
                    x = b.label[v];
                    c = (int)(a.pend[v] & 1023u);
                    s = b.off[v];
                    e = b.off[v + 1];
                    if (e - s > kLoopShort) e = s;  // in pieces
                }
                long long in_c = 0, out_a = 0;
                int dv = 0;
                mover_arcs(x, c, s, e, lane & (kGroup - 1), kGroup, in_c, out_a, dv);
                mover_done(kGroup, v, x, c, in_c, out_a, dv);
                if ((lane & (kGroup - 1)) == 0) rd += (unsigned long long)(e - s);
            }
            if (t < a.iters) {
                auto mark = [&](int64_t s, int64_t e, int first, int step) {
                    for (int64_t j0 = s + first; j0 < e; j0 += 4 * step) {
                        int u[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) u[q] = j0 + q * step < e ? __ldg(b.col + j0 + q * step) : -1;
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (u[q] >= 0) b.stamp[u[q]] = t + 1;
                    }
                };
                for (int q = ww; q < nwp; q += ms) {
                    const int2 y = a.wpiece[q];
                    const int64_t s = b.off[y.x] + y.y;
                    mark(s, min((long long)b.off[y.x + 1], (long long)s + kLoopPiece), lane, 32);
                }
                for (int i = ww * kRows + lane / kGroup; i < nwin; i += ms * kRows) {
                    const int v = a.win[i];
                    const int64_t s = b.off[v], e = b.off[v + 1];
                    if ((lane & (kGroup - 1)) == 0) b.stamp[v] = t + 1;
                    if (e - s <= kLoopShort) mark(s, e, lane & (kGroup - 1), kGroup);
                }
            }
            block_sums((unsigned long long)dcut, rd, 0, 0, [&](int j, unsigned long long s) {
                if (j == 0) atomicAdd(&b.cnt->cut_arcs, s);  // mod 2^64
                else atomicAdd(&cn->arcs_upd, s);
            });
            for (int p = threadIdx.x; p < k; p += kLoopThreads) {  // (a barrier in block_sums)
                if (s_vc[p]) atomicAdd(&b.vc[p], (unsigned long long)s_vc[p]);
                if (s_in[p]) atomicAdd(&b.intra[p], (unsigned long long)s_in[p]);
                s_vc[p] = s_in[p] = 0;
            }
        }
        if (!grid_sync(ctl, a.polls, 46)) return;
    }
    // ---- the last iteration's movers take their labels; the run's result ----
    if (t > 1) {
        const int n = __ldcg(&a.cnt[(t + 1) & 1].nmov);
        for (int i = B * kLoopThreads + threadIdx.x; i < n; i += G * kLoopThreads) {
            const int v = a.mov[i];
            b.label[v] = (int)(a.pend[v] & 1023u);
        }
    }
    if (B == 0 && threadIdx.x == 0) {
        if (bad0) ctl->error = 1;
        ctl->mode = a.mode;
        ctl->prev_cut = prev_cut;
        ctl->conv = conv;
        ctl->iters_run = iters;
        ctl->stop_reason = reason;
        ctl->stop_now = reason;
        ctl->stopped = reason != 0;
        ctl->pull = 0;
    }
}

int grid_blocks(const dmolp_ctx *c, int npos, int per_block) {
    return std::min(c->num_sms, std::max(8, (npos + per_block - 1) / per_block));
}

// All blocks are resident: at most one per SM, a cooperative launch.
template <typename K, typename A0, typename... A>
void launch_coop(dmolp_ctx *c, K kernel, int grid, int threads, size_t smem, A0 a0, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a0, args...);
    if (e != cudaSuccess && c->launch_error == cudaSuccess) c->launch_error = e;  // reported by the entry point
    c->launches += 1;
}

}  // namespace

void loop_order(dmolp_ctx *c) {
    Buffers &b = c->b;
    OrderArgs a;
    a.off = b.off;
    a.ball = b.ball;
    a.buf[0] = reinterpret_cast<int2 *>(b.dlkey);
    a.buf[1] = reinterpret_cast<int2 *>(b.dtkey);
    a.first = b.cand;
    a.last = b.bv;
    a.asc = b.lpasc;
    a.desc = b.lpdesc;
    a.blk = b.lpblk;
    a.npos = c->nb[0] + c->nb[1] + c->nb[2];
    a.npass = std::max(1, (c->dbits + 7) / 8);
    a.ctl = b.ctrl;
    a.polls = c->wait_polls;
    launch_coop(c, k_loop_order, grid_blocks(c, a.npos, kLoopBlockV), kOrderThreads, 0, a);
}

void loop_run(dmolp_ctx *c, const LpLaunch &L, int iters) {
    Buffers &b = c->b;
    LoopArgs a;
    a.ord[0] = b.lpasc;
    a.ord[1] = b.lpdesc;
    a.lab[0] = reinterpret_cast<int16_t *>(b.bown);
    a.lab[1] = reinterpret_cast<int16_t *>(b.bnew);
    a.blk = b.lpblk;
    a.pend = reinterpret_cast<uint32_t *>(b.active[0]);
    a.win = b.win[0];
    a.big = b.win[1];
    a.mov = b.mov;
    a.wpiece = b.lppiece;
    a.mpiece = b.lppiece + loop_pieces(c->narcs);
    a.cnt = reinterpret_cast<LoopCnt *>(b.lpcnt);
    a.narcs = (long long)c->narcs;
    a.npos = c->nb[0] + c->nb[1] + c->nb[2];
    a.nv = (int)c->nv;
    a.k = L.k;
    a.eff = L.eff;
    a.mode = L.mode;
    a.iters = iters;
    a.kept = c->counts_kept ? 1 : 0;
    a.hubs = c->nb[2] > 0 ? 1 : 0;
    a.polls = c->wait_polls;
    static_assert(2 * sizeof(LoopCnt) <= kLoopCntBytes, "the counters fit their buffer");
    cudaMemsetAsync(b.lpcnt, 0, kLoopCntBytes, c->stream);
    launch_coop(c, k_lp_loop, grid_blocks(c, a.npos, kLoopBlockV), kLoopThreads, loop_smem(L.k), b, a);
}

void loop_prepare() {
    cudaFuncSetAttribute(k_lp_loop, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)loop_smem(DMOLP_MAX_K));
}

}  // namespace dmolp
