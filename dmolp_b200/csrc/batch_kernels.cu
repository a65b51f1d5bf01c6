// Batched boundary label propagation: thousands of independent partition instances in a few persistent
// launches, replayed from a captured CUDA graph.
//
// Each instance is one graph of the batch (its vertices are a contiguous range of the batch's union CSR)
// with its own part count k <= 64.  A team of C CTAs -- one CTA, or a thread-block cluster of 2 to 16 --
// runs the whole phase-2 loop of src/phase2/phase2.cpp:256-449 on it: penalties, candidate marking, boundary
// test, per-label window selection, decisions, incremental cut / balance update, stopping rules, with a
// barrier of the team between the steps.  The per-instance arithmetic is the single-graph path's: the same
// penalties (warp_penalties), the same selection keys (degree ascending, or max-degree minus degree when
// RE > 1, then the vertex's id within its graph), the same decision rule and tie order, so every instance
// ends bit-identical to a single-graph run of the same graph and labels.
//
// Why teams: an iteration is a chain of short steps, each bound by the latency of its gathers (L2, ~700
// cycles), so a graph's time is its vertices per thread times that chain.  With one CTA per graph a batch
// took as long as its largest graph on one SM while the others idled; the host gives each graph CTAs in
// proportion to its share of the batch (batch_cabi.cu, team_sizes).  Phase 2 of 64 mixed graphs (2.2 M
// vertices, 27 M arcs, the largest 195 K vertices): 98 -> 4.3 ms; of 512 graphs of 1 K to 10 K vertices,
// where most teams are one CTA: 6.7 -> 3.0 ms, from the three points below.
//
// Counters the team shares (list lengths, the cut's change) live in the first CTA's shared memory and are
// reached through distributed shared memory; histograms and part counts are kept per CTA and summed over
// the team where they are read.  Work inside a team is scheduled per warp: a warp takes 32 list entries;
// rows of at most TD arcs are walked by their own lane (eight ids in flight), longer rows by the whole warp,
// one after another.
//
//  * Candidates are not listed: marking stores stamps (no atomics), and one coalesced scan over the graph's
//    vertices does candidacy, the boundary test and the first histogram of the selection.
//  * The selection is an MSD radix select with 6-bit digits over records (part, key) of 8 bytes, so no pass
//    gathers labels or degrees; each pass scatters the records that stay open and counts their next digit.
//  * Decisions of symmetric graphs with at most 32 scored labels read kept label counts (16 bits per label
//    and vertex, built by the first statistics pass and updated from the movers): a vertex costs one row of
//    at most 64 bytes instead of a gather per arc.  Other graphs recount from the arcs.
//
// Block size NT, the thread-row limit TD and the number of resident CTAs per SM are the autotuned shape.
#include <cooperative_groups.h>

#include <cfloat>

#include "batch.cuh"
#include "lp_device.cuh"
#include "team.cuh"

namespace dmolp {
namespace batch {
namespace {

constexpr int kCountRow = 32;  // statistics: rows of at most this many arcs are counted by one lane
constexpr int kScanU = 4;      // vertices per lane and step of the boundary scan

// Counters the team shares (in the first CTA's shared memory), by iteration parity.
struct Shared {
    int nbnd, nwin, nmov;
    int nact[kMaxPass];
    unsigned long long te_cand, te_sel;
    long long dcut;
};

template <int NT>
struct Smem {
    long long vc[kBatchMaxK], intra[kBatchMaxK];    // this CTA's share: the sum over the team is the count
    long long tvc[kBatchMaxK], tintra[kBatchMaxK];  // the sums at the iteration's start
    double tpen[kBatchMaxK], RE[kBatchMaxK];
    int bcnt[kBatchMaxK], need[kBatchMaxK], below[kBatchMaxK], keep[kBatchMaxK];
    union {
        int hist[2][kBatchMaxK * kDigits];  // zero between selections
        unsigned int bytes[8][NT];          // statistics: byte counters of 32 labels per thread
    };
    int whist[NT / 32][kBatchMaxK];
    Shared sh[2];
    long long cut_arcs;
    int bad, inst;
    unsigned long long arcs, visits;
};

__device__ __forceinline__ void warp_sum_into(long long x, long long *dst) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(DMOLP_FULL_MASK, x, o);
    if ((threadIdx.x & 31) == 0 && x) atomicAdd((unsigned long long *)dst, (unsigned long long)x);
}

// Label counts and same-label / cut arcs of the instance's current labels (phase2.cpp:55-117, 214-253), each
// CTA's share into its own counters; with keep_counts also the label counts of every vertex's row.  The
// team's barriers before (zeroed counters) and after are the caller's.
template <int NT, int TD, typename Tm>
__device__ void full_stats(const Args &a, const Inst &I, const Tm &tm, Smem<NT> &sm, bool keep_counts, int eff) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int words = I.cstride >> 1;  // 32-bit words of a count row
    unsigned int *const cw = reinterpret_cast<unsigned int *>(a.cnt + I.cbase);
    unsigned char *const mine = reinterpret_cast<unsigned char *>(&sm.bytes[0][threadIdx.x]);
    constexpr int kByteRow = NT * 4;  // bytes between a thread's consecutive counter words
    long long cut = 0;
    int bad = 0;
    visit(a.off, tm, I.nv, [&](int i) { return (int)I.vbase + i; },
          [&](int, int64_t s, int64_t e) { return e - s > (keep_counts ? kCountRow : TD); },
          [&](bool act, int v, int64_t s, int64_t e) {
              if (!act) return;
              const int lv = a.label[v];
              if ((unsigned)lv >= (unsigned)I.k) {
                  bad = 1;
                  return;
              }
              if (keep_counts)
#pragma unroll
                  for (int w = 0; w < 8; ++w) sm.bytes[w][threadIdx.x] = 0u;
              int same = 0;
              const int deg = (int)(e - s);
              for (int j = 0; j < deg; j += 8) {
                  int l[8];
#pragma unroll
                  for (int q = 0; q < 8; ++q) l[q] = j + q < deg ? a.label[__ldg(a.col + s + j + q)] : -1;
#pragma unroll
                  for (int q = 0; q < 8; ++q) {
                      same += l[q] == lv;
                      if (keep_counts && (unsigned)l[q] < (unsigned)eff) mine[(l[q] >> 2) * kByteRow + (l[q] & 3)] += 1;
                  }
              }
              atomicAdd((unsigned long long *)&sm.vc[lv], 1ull);
              if (same) atomicAdd((unsigned long long *)&sm.intra[lv], (unsigned long long)same);
              cut += deg - same;
              a.ndiff[v] = deg - same;
              if (keep_counts) {
                  uint2 *const row = reinterpret_cast<uint2 *>(cw + (size_t)(v - (int)I.vbase) * words);
                  for (int w = 0; w < words / 2; ++w) {  // four byte counters -> four 16-bit counts
                      const unsigned int x = sm.bytes[w][threadIdx.x];
                      row[w] = make_uint2(__byte_perm(x, 0, 0x4140), __byte_perm(x, 0, 0x4342));
                  }
              }
          },
          [&](int v, int64_t s, int64_t e) {
              const int lv = a.label[v];
              int *h = sm.whist[wib];
              if (keep_counts) {
                  h[lane] = 0;
                  __syncwarp();
              }
              int same = 0;
              warp_row_wide(a.col, s, e, lane, [&](int u) { return a.label[u]; }, [&](int, int lu) {
                  same += lu == lv;
                  if (keep_counts && (unsigned)lu < (unsigned)eff) atomicAdd(&h[lu], 1);
              }, [] { return false; });
              for (int o = 16; o > 0; o >>= 1) same += __shfl_xor_sync(DMOLP_FULL_MASK, same, o);
              const int diff = (int)(e - s) - same;
              if ((unsigned)lv >= (unsigned)I.k) {
                  bad = 1;
              } else if (lane == 0) {
                  atomicAdd((unsigned long long *)&sm.vc[lv], 1ull);
                  if (same) atomicAdd((unsigned long long *)&sm.intra[lv], (unsigned long long)same);
                  cut += diff;
                  a.ndiff[v] = diff;
              }
              if (keep_counts) {
                  __syncwarp();
                  if (lane < words)
                      cw[(size_t)(v - (int)I.vbase) * words + lane] =
                          (unsigned int)h[2 * lane] | ((unsigned int)h[2 * lane + 1] << 16);
                  __syncwarp();
              }
          });
    warp_sum_into(cut, tm.first(&sm.cut_arcs));
    if (__any_sync(DMOLP_FULL_MASK, bad) && lane == 0) *tm.first(&sm.bad) = 1;
}

template <int NT, int TD, typename Tm>
__device__ void run_instance(const Args &a, const int ii, const Tm &tm, Smem<NT> &sm) {
    const Inst I = a.inst[ii];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int k = I.k, vb = (int)I.vbase;
    const int eff = a.cap == DMOLP_LP_CAP_FULL ? k : (k < 32 ? k : 32);
    const bool counts = I.cstride > 0 && eff <= 32;  // kept label counts (symmetric, 16-bit degrees)
    const int words = I.cstride >> 1;
    unsigned int *const cw = reinterpret_cast<unsigned int *>(a.cnt + I.cbase);
    const int stamp0 = *a.stamp_base;
    uint64_t *const rec[2] = {a.rec0 + I.vbase, a.rec1 + I.vbase};
    int32_t *const win[2] = {a.l_win0 + I.vbase, a.l_win1 + I.vbase};
    int32_t *const mov = a.l_bnd + I.vbase;
    const int kbits = I.dbits + I.ibits;
    const int npass = (kbits + kDigitBits - 1) / kDigitBits > 0 ? (kbits + kDigitBits - 1) / kDigitBits : 1;
    const int top = npass * kDigitBits;
    const bool packed = kbits <= kOwnShift;
    const uint64_t idmask = (uint64_t(1) << I.ibits) - 1;
    // the part of a record (its label does not change before the movers apply)
    auto part_of = [&](uint64_t r) {
        return packed ? (int)(r >> kOwnShift) : a.label[vb + (int)(r & idmask)];
    };

    for (int p = threadIdx.x; p < kBatchMaxK; p += NT) sm.vc[p] = sm.intra[p] = 0;
    if (threadIdx.x == 0) {
        sm.cut_arcs = 0;
        sm.bad = 0;
        sm.arcs = sm.visits = 0;
    }
    if (threadIdx.x < 2) sm.sh[threadIdx.x] = Shared();
    tm.sync();
    full_stats<NT, TD>(a, I, tm, sm, counts, eff);
    tm.sync();
    for (int i = threadIdx.x; i < 2 * kBatchMaxK * kDigits; i += NT) (&sm.hist[0][0])[i] = 0;  // (was byte counters)
    long long cut_arcs = *tm.first(&sm.cut_arcs);
    Out o;
    o.edge_cut = cut_arcs >> 1;
    o.te = o.arcs = o.visits = 0;
    o.iterations = o.stop_reason = o.changes = 0;
    o.status = (*tm.first(&sm.bad) || (cut_arcs & 1)) ? DMOLP_ERR_BAD_LABELS : DMOLP_OK;
    const int max_iter = a.mode == DMOLP_LP_MODE_REF ? kMaxIter : a.iters;
    long long prev_cut = o.edge_cut;
    int conv = 0;
    unsigned long long te_prev_next = (unsigned long long)I.narcs;
    int nprev = I.nv;
    unsigned long long arcs = 0, visits = 0;
    for (int t = 1; o.status == DMOLP_OK && t <= max_iter; ++t) {
        const int st = stamp0 + t;
        Shared *const sh = tm.first(&sm.sh[t & 1]);
        // ---- penalties (phase2.cpp:158-209), by every CTA from the team's counts ----
        for (int p = threadIdx.x; p < k; p += NT) {
            long long x = 0, y = 0;
            for (int r = 0; r < tm.size(); ++r) {
                x += *tm.at(&sm.vc[p], r);
                y += *tm.at(&sm.intra[p], r);
            }
            sm.tvc[p] = x;
            sm.tintra[p] = y;
            sm.bcnt[p] = 0;
        }
        __syncthreads();
        if (wib == 0)
            warp_penalties(k, [&](int p) { return sm.tvc[p]; }, [&](int p) { return sm.tintra[p] / 2; }, a.logtab[t],
                           sm.RE, sm.tpen, nullptr);
        const unsigned long long te_prev = te_prev_next;
        // ---- candidates = previous window and its neighbours (gpu_lp_boundary.cu:196-214) ----
        if (t > 1) {
            const int32_t *prev = win[(t - 1) & 1];
            visit(a.off, tm, nprev, [&](int i) { return prev[i]; }, [&](int, int64_t s, int64_t e) { return e - s > TD; },
                  [&](bool act, int v, int64_t s, int64_t e) {
                      if (!act) return;
                      a.cstamp[v] = st;
                      const int deg = (int)(e - s);
                      for (int j = 0; j < deg; j += 8) {
                          int u[8];
#pragma unroll
                          for (int q = 0; q < 8; ++q) u[q] = j + q < deg ? __ldg(a.col + s + j + q) : -1;
#pragma unroll
                          for (int q = 0; q < 8; ++q)
                              if (u[q] >= 0) a.cstamp[u[q]] = st;
                      }
                      ++visits;
                      arcs += (unsigned long long)deg;
                  },
                  [&](int v, int64_t s, int64_t e) {
                      if (lane == 0) {
                          a.cstamp[v] = st;
                          ++visits;
                          arcs += (unsigned long long)(e - s);
                      }
                      warp_row(a.col, s, e, lane, [&](int u) { a.cstamp[u] = st; }, [] { return false; });
                  });
            tm.sync();
        } else {
            __syncthreads();  // the penalties
        }
        // ---- boundary test over all vertices: a candidate with a neighbour of another label
        //      (gpu_lp_boundary.cu:216-236), i.e. ndiff > 0; its record and first digit ----
        if (tm.is_first() && threadIdx.x == 0) sm.sh[(t + 1) & 1] = Shared();  // last read before this barrier
        {
            unsigned long long tec = 0;
            for (int i0 = tm.warp() * 32 * kScanU; i0 < I.nv; i0 += tm.threads() * kScanU) {
                int deg[kScanU], nd[kScanU], own[kScanU];
                bool isb[kScanU];
#pragma unroll
                for (int q = 0; q < kScanU; ++q) {
                    const int i = i0 + q * 32 + lane;
                    const bool in = i < I.nv;
                    const int v = vb + (in ? i : 0);
                    isb[q] = in && (t == 1 || a.cstamp[v] == st);
                    deg[q] = (int)(a.off[v + 1] - a.off[v]);
                    nd[q] = a.ndiff[v];
                    own[q] = a.label[v];
                }
                unsigned m[kScanU];
                int tot = 0;
#pragma unroll
                for (int q = 0; q < kScanU; ++q) {
                    if (isb[q]) {
                        tec += (unsigned long long)deg[q];
                        ++visits;
                    }
                    isb[q] = isb[q] && nd[q] > 0;
                    m[q] = __ballot_sync(DMOLP_FULL_MASK, isb[q]);
                    tot += __popc(m[q]);
                }
                int base = 0;
                if (lane == 0 && tot) base = atomicAdd(&sh->nbnd, tot);
                base = __shfl_sync(DMOLP_FULL_MASK, base, 0);
#pragma unroll
                for (int q = 0; q < kScanU; ++q) {
                    if (isb[q]) {
                        const int p = own[q];
                        const uint64_t dk = sm.RE[p] > 1.0 ? (uint64_t)(I.maxdeg - deg[q]) : (uint64_t)deg[q];
                        const uint64_t key = (dk << I.ibits) | (uint64_t)(i0 + q * 32 + lane);
                        rec[0][base + __popc(m[q] & ((1u << lane) - 1))] =
                            packed ? key | ((uint64_t)p << kOwnShift) : key;
                        atomicAdd(&sm.bcnt[p], 1);
                        atomicAdd(&sm.hist[0][p * kDigits + (int)((key >> (top - kDigitBits)) & (kDigits - 1))], 1);
                    }
                    base += __popc(m[q]);
                }
            }
            tec = warp_sum_u64(tec);
            if (lane == 0 && tec) atomicAdd(&sh->te_cand, tec);
        }
        tm.sync();
        // ---- per label keep ceil(e^(-t/5) * n_p) (gpu_lp_boundary.cu:238-300) ----
        {
            const double ratio = a.ratiotab[t];
            for (int p = threadIdx.x; p < k; p += NT) {
                int n = 0;
                for (int r = 0; r < tm.size(); ++r) n += *tm.at(&sm.bcnt[p], r);
                const int m = (int)ceil(__dmul_rn(ratio, (double)n));
                sm.need[p] = m > n ? n : m;
            }
        }
        __syncthreads();
        int32_t *const wout = win[t & 1];
        int nlist = sh->nbnd;
        for (int pass = 0; pass < npass; ++pass) {
            const int shift = top - kDigitBits * (pass + 1);
            cut_digit(tm, k, sm.hist[pass & 1], sm.need, sm.below, sm.keep);
            tm.sync();
            const bool open = any_open(k, sm.keep);
            // records below the digit are selected; records on it stay, counted by their next digit
            for (int i = threadIdx.x; i < k * kDigits; i += NT) sm.hist[pass & 1][i] = 0;
            const uint64_t *const list = rec[pass & 1];
            uint64_t *const nxt = rec[(pass + 1) & 1];
            for (int i0 = tm.warp() * 32; i0 < nlist; i0 += tm.threads()) {
                const int i = i0 + lane;
                bool take = false, keep = false;
                uint64_t r = 0;
                int p = 0;
                if (i < nlist) {
                    r = list[i];
                    p = part_of(r);
                    const int d = (int)((r >> shift) & (kDigits - 1));
                    take = d < sm.below[p];
                    keep = d == sm.keep[p];
                }
                const int ws = warp_push(&sh->nwin, take);
                if (take) wout[ws] = vb + (int)(r & idmask);
                const int ks = warp_push(&sh->nact[pass], keep);
                if (keep) {
                    nxt[ks] = r;
                    atomicAdd(&sm.hist[(pass + 1) & 1][p * kDigits + (int)((r >> (shift - kDigitBits)) & (kDigits - 1))],
                              1);
                }
            }
            tm.sync();
            if (!open) break;
            nlist = sh->nact[pass];
        }
        const int nwin = sh->nwin;
        // ---- decisions for the window (boundaryLPKernel_unified, gpu_lp_boundary.cu:327-427) ----
        unsigned long long tes = 0;
        if (counts) {
            for (int i0 = tm.warp() * 32; i0 < nwin; i0 += tm.threads()) {
                const int i = i0 + lane;
                int nl = -1, v = 0;
                if (i < nwin) {
                    v = wout[i];
                    const int own = a.label[v];
                    tes += (unsigned long long)(a.off[v + 1] - a.off[v]);
                    ++visits;
                    const uint4 *const row = reinterpret_cast<const uint4 *>(cw + (size_t)(v - vb) * words);
                    double best = -DBL_MAX;
                    int bkey = 0x7fffffff, blab = -1, own_cnt = -1;
                    for (int c0 = 0; c0 < eff; c0 += 8) {
                        const uint4 x = row[c0 >> 3];
                        const unsigned int w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const int c = c0 + q;
                            const int n = (int)((w[q >> 1] >> (16 * (q & 1))) & 0xffffu);
                            if (c == own) own_cnt = n;
                            if (c < eff && (n > 0 || own >= eff)) {
                                const double sc = n > 0 ? __dmul_rn((double)n, sm.tpen[c]) : 0.0;
                                const int key = tiekey(c);
                                if (better(sc, key, best, bkey)) {
                                    best = sc;
                                    bkey = key;
                                    blab = c;
                                }
                            }
                        }
                    }
                    const double own_raw = own < eff ? (double)own_cnt : -1e300;
                    if (blab >= 0 && best > own_raw && blab != own) nl = blab;
                }
                const int slot = warp_push(&sh->nmov, nl >= 0);
                if (nl >= 0) {
                    a.newlab[v] = nl;
                    mov[slot] = v;
                }
            }
        } else {
            int *h = sm.whist[wib];
            visit(a.off, tm, nwin, [&](int i) { return wout[i]; },
                  [&](int v, int64_t s, int64_t e) { return e - s > TD || a.label[v] >= eff; },
                  [&](bool act, int v, int64_t s, int64_t e) {
                      int nl = -1;
                      if (act) {
                          const int own = a.label[v];
                          const int deg = (int)(e - s);
                          tes += (unsigned long long)deg;
                          arcs += (unsigned long long)deg;
                          ++visits;
                          int l[TD];
#pragma unroll
                          for (int j = 0; j < TD; ++j) l[j] = j < deg ? a.label[__ldg(a.col + s + j)] : -1;
                          int own_cnt = 0;
                          double best = -DBL_MAX;
                          int bkey = 0x7fffffff, blab = -1;
#pragma unroll
                          for (int j = 0; j < TD; ++j) {
                              own_cnt += (l[j] == own);
                              const int c = l[j];
                              if ((unsigned)c < (unsigned)eff) {
                                  int cnt = 0;
#pragma unroll
                                  for (int q = 0; q < TD; ++q) cnt += (l[q] == c);
                                  const double sc = __dmul_rn((double)cnt, sm.tpen[c]);
                                  const int key = tiekey(c);
                                  if (better(sc, key, best, bkey)) {
                                      best = sc;
                                      bkey = key;
                                      blab = c;
                                  }
                              }
                          }
                          if (blab >= 0 && best > (double)own_cnt && blab != own) nl = blab;
                      }
                      const int slot = warp_push(&sh->nmov, nl >= 0);
                      if (nl >= 0) {
                          a.newlab[v] = nl;
                          mov[slot] = v;
                      }
                  },
                  [&](int v, int64_t s, int64_t e) {
                      const int own = a.label[v];
                      for (int c = lane; c < eff; c += 32) h[c] = 0;
                      __syncwarp();
                      warp_row_wide(a.col, s, e, lane, [&](int u) { return a.label[u]; }, [&](int, int lu) {
                          if ((unsigned)lu < (unsigned)eff) atomicAdd(&h[lu], 1);
                      }, [] { return false; });
                      __syncwarp();
                      double best;
                      int blab;
                      warp_argmax(eff, sm.tpen, lane, [&](int c) { return h[c]; }, best, blab);
                      const double own_raw = (unsigned)own < (unsigned)eff ? (double)h[own] : -1e300;
                      __syncwarp();
                      if (lane == 0) {
                          tes += (unsigned long long)(e - s);
                          arcs += (unsigned long long)(e - s);
                          ++visits;
                          const int nl = best > own_raw ? blab : own;
                          if (nl != own) {
                              a.newlab[v] = nl;
                              mov[atomicAdd(&sh->nmov, 1)] = v;
                          }
                      }
                  });
        }
        tes = warp_sum_u64(tes);
        if (lane == 0 && tes) atomicAdd(&sh->te_sel, tes);
        tm.sync();
        const int nmov = sh->nmov;
        // ---- incremental cut / balance / count update from the movers (symmetric graphs) ----
        if (I.symmetric && nmov > 0) {
            long long dcut = 0;
            // cut / intra counts, and the differently-labelled neighbour counts: arc (u,v) seen from u, arc
            // (v,u) from v when u stays (a moving u updates v's count from its own row); the kept counts of u
            // lose v's old label and gain its new one.  a0 -> c: v's labels; lo, nu: u's label and its new one
            auto upd = [&](int u, int lo, int nu, int a0, int c, long long &dc, int &in_c, int &out_a, int &dv) {
                const int ln = nu >= 0 ? nu : lo;
                const int w = nu >= 0 ? 1 : 2;
                dc += w * ((int)(c != ln) - (int)(a0 != lo));
                in_c += w * (int)(c == ln);
                out_a += w * (int)(a0 == lo);
                const int du = (int)(ln != c) - (int)(lo != a0);
                if (du) atomicAdd(&a.ndiff[u], du);
                if (nu < 0) dv += (int)(c != lo) - (int)(a0 != lo);
                if (counts) {  // 16-bit halves: the sums end non-negative, so borrows between them cancel
                    unsigned int *const row = cw + (size_t)(u - vb) * words;
                    const unsigned int minus = (unsigned int)-(1 << (16 * (a0 & 1))), plus = 1u << (16 * (c & 1));
                    if ((a0 >> 1) == (c >> 1)) {
                        atomicAdd(&row[c >> 1], minus + plus);
                    } else {
                        if (a0 < eff) atomicAdd(&row[a0 >> 1], minus);
                        if (c < eff) atomicAdd(&row[c >> 1], plus);
                    }
                }
            };
            visit(a.off, tm, nmov, [&](int i) { return mov[i]; }, [&](int, int64_t s, int64_t e) { return e - s > TD; },
                  [&](bool act, int v, int64_t s, int64_t e) {
                      if (!act) return;
                      const int a0 = a.label[v], c = a.newlab[v], deg = (int)(e - s);
                      int in_c = 0, out_a = 0, dv = 0;
                      for (int j = 0; j < deg; j += 4) {
                          int u[4], lo[4], nu[4];
#pragma unroll
                          for (int q = 0; q < 4; ++q) u[q] = j + q < deg ? __ldg(a.col + s + j + q) : -1;
#pragma unroll
                          for (int q = 0; q < 4; ++q) {
                              lo[q] = u[q] >= 0 ? a.label[u[q]] : 0;
                              nu[q] = u[q] >= 0 ? a.newlab[u[q]] : 0;
                          }
#pragma unroll
                          for (int q = 0; q < 4; ++q)
                              if (u[q] >= 0) upd(u[q], lo[q], nu[q], a0, c, dcut, in_c, out_a, dv);
                      }
                      if (dv) atomicAdd(&a.ndiff[v], dv);
                      arcs += (unsigned long long)deg;
                      ++visits;
                      atomicAdd((unsigned long long *)&sm.vc[a0], (unsigned long long)-1ll);
                      atomicAdd((unsigned long long *)&sm.vc[c], 1ull);
                      if (in_c) atomicAdd((unsigned long long *)&sm.intra[c], (unsigned long long)in_c);
                      if (out_a) atomicAdd((unsigned long long *)&sm.intra[a0], (unsigned long long)-(long long)out_a);
                  },
                  [&](int v, int64_t s, int64_t e) {
                      const int a0 = a.label[v], c = a.newlab[v];
                      long long dc = 0;
                      int in_c = 0, out_a = 0, dv = 0;
                      warp_row(a.col, s, e, lane,
                               [&](int u) { upd(u, a.label[u], a.newlab[u], a0, c, dc, in_c, out_a, dv); },
                               [] { return false; });
                      for (int o2 = 16; o2 > 0; o2 >>= 1) {
                          in_c += __shfl_xor_sync(DMOLP_FULL_MASK, in_c, o2);
                          out_a += __shfl_xor_sync(DMOLP_FULL_MASK, out_a, o2);
                          dv += __shfl_xor_sync(DMOLP_FULL_MASK, dv, o2);
                      }
                      dcut += dc;
                      if (lane == 0) {
                          if (dv) atomicAdd(&a.ndiff[v], dv);
                          arcs += (unsigned long long)(e - s);
                          ++visits;
                          atomicAdd((unsigned long long *)&sm.vc[a0], (unsigned long long)-1ll);
                          atomicAdd((unsigned long long *)&sm.vc[c], 1ull);
                          if (in_c) atomicAdd((unsigned long long *)&sm.intra[c], (unsigned long long)in_c);
                          if (out_a) atomicAdd((unsigned long long *)&sm.intra[a0], (unsigned long long)-(long long)out_a);
                      }
                  });
            warp_sum_into(dcut, &sh->dcut);
        }
        tm.sync();
        // ---- movers take their labels ----
        for (int i = tm.thread(); i < nmov; i += tm.threads()) {
            const int v = mov[i];
            a.label[v] = a.newlab[v];
            a.newlab[v] = -1;
        }
        // ---- stopping rules (phase2.cpp:305-415), by every thread alike ----
        bool stats = true;
        int stop = 0;
        if (nwin == 0) {
            stats = false;
            if (a.mode == DMOLP_LP_MODE_REF) stop = 1;
        } else if (nmov == 0 && a.mode == DMOLP_LP_MODE_REF) {
            stats = false;
            stop = 2;
        }
        long long ca = cut_arcs + sh->dcut;
        const unsigned long long te_cand = sh->te_cand, te_sel = sh->te_sel;
        if (stats && !I.symmetric) {  // no reverse arcs to update from: recount
            for (int p = threadIdx.x; p < k; p += NT) sm.vc[p] = sm.intra[p] = 0;
            if (threadIdx.x == 0) sm.cut_arcs = 0;
            tm.sync();
            full_stats<NT, TD>(a, I, tm, sm, false, eff);
            tm.sync();
            ca = *tm.first(&sm.cut_arcs);
        }
        if (stats) {
            if (ca & 1) {
                o.status = DMOLP_ERR_BAD_LABELS;
                stop = 4;
            } else {
                const long long cur = ca >> 1;
                const double delta =
                    prev_cut > 0 ? fabs(__ddiv_rn((double)(cur - prev_cut), (double)prev_cut)) : 1.0;
                if (delta < 0.03) ++conv;
                else conv = 0;
                prev_cut = cur;
                if (a.mode == DMOLP_LP_MODE_REF && conv >= 10) stop = 3;
            }
            cut_arcs = ca;
        }
        o.te += te_prev + te_cand + te_sel + (stats ? (unsigned long long)I.narcs : 0ull);
        o.changes += nmov;
        o.iterations = t;
        te_prev_next = te_sel;
        nprev = nwin;
        if (stop) {
            o.stop_reason = stop;
            break;
        }
    }
    arcs = warp_sum_u64(arcs);
    visits = warp_sum_u64(visits);
    if (lane == 0) {
        atomicAdd(tm.first(&sm.arcs), arcs);
        atomicAdd(tm.first(&sm.visits), visits);
    }
    tm.sync();
    if (tm.is_first()) {
        o.edge_cut = prev_cut;
        o.arcs = sm.arcs;
        o.visits = sm.visits;
        if (threadIdx.x == 0) a.out[ii] = o;
        long long *cnt = a.counts + (size_t)ii * 2 * kBatchMaxK;
        for (int p = threadIdx.x; p < kBatchMaxK; p += NT) {
            long long x = 0, y = 0;
            for (int r = 0; p < k && r < tm.size(); ++r) {
                x += *tm.at(&sm.vc[p], r);
                y += *tm.at(&sm.intra[p], r);
            }
            cnt[p] = x;
            cnt[kBatchMaxK + p] = y / 2;
        }
    }
    tm.sync();  // no CTA leaves, or starts on another graph, while its counters are read
}

// One CTA per graph: persistent CTAs take the graphs order[0, n) from a queue.
template <int NT, int TD>
__global__ void __launch_bounds__(NT, 1024 / NT) k_batch_lp(Args a, const int32_t *order, int n) {
    __shared__ Smem<NT> sm;
    const CtaTeam<NT> tm;
    for (;;) {
        if (threadIdx.x == 0) sm.inst = atomicAdd(a.next, 1);
        __syncthreads();
        const int q = sm.inst;
        __syncthreads();  // every thread has read it before it is rewritten
        if (q >= n) break;
        run_instance<NT, TD>(a, order[q], tm, sm);
    }
}

// One cluster per graph: cluster c runs order[c].
template <int NT, int TD>
__global__ void __launch_bounds__(NT, 1024 / NT) k_batch_lp_team(Args a, const int32_t *order) {
    __shared__ Smem<NT> sm;
    const ClusterTeam<NT> tm;
    run_instance<NT, TD>(a, order[blockIdx.x / tm.size()], tm, sm);
}

__global__ void k_batch_begin(int *next, int *stamp_base) {
    *next = 0;
    *stamp_base += kStampStride;
}

// ------------------------------------------------------------------------------------ upload
// The row of arc j: the last v with off[v] <= j.
__device__ __forceinline__ int64_t row_of(const int64_t *off, int64_t nv, int64_t j) {
    int64_t lo = 0, hi = nv;  // off[lo] <= j < off[hi]
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (off[mid] <= j) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The instance of vertex v: the last one whose first vertex is <= v (empty instances before it share it).
__device__ __forceinline__ int inst_of(const Inst *inst, int ninst, int64_t v) {
    int lo = 0, hi = ninst;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (inst[mid].vbase <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The three passes of an upload's check run over all arcs (or vertices) of the batch alike, whatever the
// graphs' sizes and degrees: each thread finds its arc's row and graph by bisection.  One block per graph
// and one thread per row, as before, took 3.9 s for one skewed graph of a million vertices.
// Local neighbour ids -> union ids, with the range check (err: 1 + an instance with a bad id).
__global__ void k_batch_ids(const int64_t *off, int32_t *col, const Inst *inst, int ninst, int64_t nv, int64_t narcs,
                            int *err) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < narcs; j += (int64_t)gridDim.x * blockDim.x) {
        const int i = inst_of(inst, ninst, row_of(off, nv, j));
        const int u = col[j];
        if ((unsigned)u >= (unsigned)inst[i].nv) atomicMax(err, i + 1);
        else col[j] = u + (int)inst[i].vbase;
    }
}

// Whether every row is strictly increasing and every arc has its reverse (bisection in the neighbour's row).
__global__ void k_batch_symmetric(const int64_t *off, const int32_t *col, Inst *inst, int ninst, int64_t nv,
                                  int64_t narcs, const int *err) {
    if (*err) return;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < narcs; j += (int64_t)gridDim.x * blockDim.x) {
        const int v = (int)row_of(off, nv, j);
        const int u = col[j];
        bool bad = j > off[v] && col[j - 1] >= u;
        if (!bad) {
            const int64_t ue = off[u + 1];
            int64_t lo = off[u], hi = ue;
            while (lo < hi) {
                const int64_t mid = (lo + hi) >> 1;
                if (col[mid] < v) lo = mid + 1;
                else hi = mid;
            }
            bad = lo >= ue || col[lo] != v;
        }
        if (bad) inst[inst_of(inst, ninst, v)].symmetric = 0;
    }
}

// Largest degree per instance (one atomic per warp where its vertices share the instance), and the list of
// rows longer than kLongRow.
__global__ void k_batch_degrees(const int64_t *off, Inst *inst, int ninst, int64_t nv, int32_t *longrow, int *nlong) {
    const int lane = threadIdx.x & 31;
    for (int64_t v0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~int64_t(31); v0 < nv;
         v0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = v0 + lane < nv ? v0 + lane : nv - 1;
        const int i = inst_of(inst, ninst, v), deg = (int)(off[v + 1] - off[v]);
        if (__all_sync(DMOLP_FULL_MASK, i == __shfl_sync(DMOLP_FULL_MASK, i, 0))) {
            const int m = __reduce_max_sync(DMOLP_FULL_MASK, deg);
            if (lane == 0) atomicMax(&inst[i].maxdeg, m);
        } else {
            atomicMax(&inst[i].maxdeg, deg);
        }
        const bool lg = v0 + lane < nv && deg > kLongRow;
        const int at = warp_push(nlong, lg);
        if (lg) longrow[at] = (int)v;
    }
}

// f(kernel, cluster kernel) for the variant (nt, td); false when there is none.
template <typename F>
bool with_variant(int nt, int td, F f) {
#define DMOLP_VARIANT(NT_, TD_)                                     \
    if (nt == NT_ && td == TD_) {                                   \
        f(k_batch_lp<NT_, TD_>, k_batch_lp_team<NT_, TD_>);         \
        return true;                                                \
    }
    DMOLP_VARIANT(256, 8) DMOLP_VARIANT(256, 16) DMOLP_VARIANT(512, 8) DMOLP_VARIANT(512, 16) DMOLP_VARIANT(1024, 8)
    DMOLP_VARIANT(1024, 16)
#undef DMOLP_VARIANT
    return false;
}

}  // namespace

int occupancy(int nt, int td) {
    int n = 0;
    cudaError_t e = cudaSuccess;
    with_variant(nt, td, [&](auto one, auto) { e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, one, nt, 0); });
    return e == cudaSuccess ? n : 0;
}

int max_team(int nt, int td) {
    int best = 1;
    with_variant(nt, td, [&](auto, auto team) {
        for (int c = kMaxTeam; c > 1 && best == 1; c >>= 1) {
            int n = 0;
            if (max_clusters(team, c, nt, &n) && n > 0) best = c;
        }
    });
    return best;
}

bool launch(const Args &a, int nt, int td, int grid, const TeamPlan &plan, const Fork &f, cudaStream_t s) {
    k_batch_begin<<<1, 1, 0, s>>>(a.next, a.stamp_base);
    return with_variant(nt, td, [&](auto one, auto team) {
        f.open(plan, s);
        const int32_t *order = a.order;
        for (int j = 0, c = kMaxTeam; c > 1; ++j, c >>= 1) {  // the largest graphs first
            if (plan.n[j] > 0) launch_cluster(team, plan.n[j], c, nt, f.stream(plan, j, s), a, order);
            order += plan.n[j];
        }
        const int n1 = plan.n[kTeamClasses - 1];
        if (n1 > 0) one<<<grid < n1 ? grid : n1, nt, 0, f.stream(plan, kTeamClasses - 1, s)>>>(a, order, n1);
        f.close(plan, s);
    });
}

void prepare(const int64_t *off, int32_t *col, Inst *inst, int ninst, int64_t nv, int64_t narcs, int *err,
             int32_t *longrow, int *nlong, int grid, cudaStream_t s) {
    if (narcs > 0) {
        k_batch_ids<<<grid, 256, 0, s>>>(off, col, inst, ninst, nv, narcs, err);
        k_batch_symmetric<<<grid, 256, 0, s>>>(off, col, inst, ninst, nv, narcs, err);
    }
    if (nv > 0) k_batch_degrees<<<grid, 256, 0, s>>>(off, inst, ninst, nv, longrow, nlong);
}

}  // namespace batch
}  // namespace dmolp
