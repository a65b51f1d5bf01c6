// Batched phase 1: the BFS / hub-seeded initial partition of every graph of a batch, a team of CTAs per graph
// (one CTA, or a cluster of 2 to 16: team.cuh, batch_cabi.cu team_sizes).
//
// A team runs phase 1 on its graph exactly as the single-graph path does (dmolp_phase1;
// src/phase1/seed.cpp:138-242, partition.cpp:323-604):
//   seeds       the first seed, then repeatedly the first unused hub (in hub order) of maximum degree that
//               lies outside the radius-2 balls of the seeds so far; stops when no hub is left
//   completion  where fewer than k seeds were found: unused hubs by degree (first in hub order on ties),
//               then other vertices by degree (lowest id)
//   growth      rounds: per part the theta frontier vertices with the smallest (degree, id) expand (an MSD
//               radix select, segmented by part), unlabelled neighbours are claimed with atomicMin over part
//               ids (lowest part wins), claimed vertices join their part's frontier and unselected ones carry
//               over; with every frontier empty, all unlabelled vertices go to the smallest part (lowest
//               index on ties)
// The hub lists and first seeds come from the host (the reference's order-dependent sort, computed per
// graph in the single-graph code's own function).  Degrees are CSR row lengths: a batch holds graphs with
// sorted, duplicate-free rows, whose line token counts equal them.
//
// What bounds it: latency.  Every step is a few dependent L2 gathers per vertex, so the time is the number
// of vertices per thread, the number of rounds and the barriers per round; hence teams, and
//  * the hub list is in descending degree order, so the next seed is the next uncovered hub after the last
//    one: one pass over the list for all seeds (each CTA walks it by itself, no barrier of the team);
//  * a round in which no part has more than theta frontier vertices -- most rounds -- selects nothing: two
//    barriers.  Otherwise the select runs over records (part, degree, id) of 8 bytes;
//  * claims are appended straight to the next frontier, one atomic per warp for up to 32 rows.
// 64 mixed graphs (2.2 M vertices, up to 84 rounds): 31.7 -> 1.7 ms; 512 graphs of 1 K to 10 K vertices:
// 2.6 -> 0.9 ms.
#include <algorithm>
#include <climits>

#include "batch.cuh"
#include "lp_device.cuh"
#include "team.cuh"

namespace dmolp {
namespace batch {
namespace {

constexpr int kP1Threads = 512;
constexpr int kP1Row = 32;  // rows of at most this many arcs are walked by one lane (a bit per claimed arc)

// Counters the team shares (in the first CTA's shared memory), by round parity.
struct P1Shared {
    int nnext, nsel;
    int nact[kMaxPass];
};

struct P1Smem {
    long long psize[kBatchMaxK];  // this CTA's share of the part sizes
    int npart[2][kBatchMaxK];     // its share of the frontier per part, by round parity
    int need[kBatchMaxK], below[kBatchMaxK], keep[kBatchMaxK];
    int hist[2][kBatchMaxK * kDigits];  // zero between selections
    int seeds[kBatchMaxK];
    unsigned long long wbest[kP1Threads / 32];
    unsigned long long cbest;  // the CTA's maximum
    P1Shared sh[2];
    int nfall, inst, idx;
    unsigned long long te;
};

__device__ __forceinline__ int deg_of(const P1Args &a, int v) { return (int)(a.off[v + 1] - a.off[v]); }

__device__ __forceinline__ bool is_seed(const P1Smem &sm, int n, int v) {
    bool s = false;
    for (int q = 0; q < n; ++q) s |= sm.seeds[q] == v;
    return s;
}

// The first hub at or after `from` that is no seed and, with `outside`, lies outside the balls; its index, or
// nh.  Every CTA finds it by itself.
__device__ int next_hub(const P1Args &a, const int32_t *hubs, int nh, int from, int vb, int nseeds, bool outside,
                        P1Smem &sm) {
    for (int b0 = from; b0 < nh; b0 += kP1Threads) {
        const int i = b0 + (int)threadIdx.x;
        bool ok = false;
        if (i < nh) {
            const int h = vb + hubs[i];
            ok = !(outside && a.cov[h]) && !is_seed(sm, nseeds, h);
        }
        if (threadIdx.x == 0) sm.idx = INT_MAX;
        if (!__syncthreads_or(ok)) continue;
        const unsigned m = __ballot_sync(DMOLP_FULL_MASK, ok);
        if (m && (threadIdx.x & 31) == 0) atomicMin(&sm.idx, i + __ffs(m) - 1);
        __syncthreads();
        const int r = sm.idx;
        __syncthreads();
        return r;
    }
    return nh;
}

// Radius-2 ball of seed s: level 1 its row, level 2 the rows of its neighbours (except s itself).
template <typename Tm>
__device__ void mark_ball(const P1Args &a, int s, const Tm &tm, unsigned long long &te) {
    const int lane = threadIdx.x & 31;
    const int64_t rs = a.off[s];
    const int deg = deg_of(a, s);
    if (tm.thread() == 0) {
        a.cov[s] = 1;
        te += (unsigned long long)deg;
    }
    visit(a.off, tm, deg, [&](int i) { return a.col[rs + i]; }, [&](int, int64_t b, int64_t e) { return e - b > kP1Row; },
          [&](bool act, int u, int64_t b, int64_t e) {
              if (!act) return;
              a.cov[u] = 1;
              if (u == s) return;
              const int n = (int)(e - b);
              te += (unsigned long long)n;
              for (int j = 0; j < n; j += 8) {
                  int x[8];
#pragma unroll
                  for (int q = 0; q < 8; ++q) x[q] = j + q < n ? __ldg(a.col + b + j + q) : -1;
#pragma unroll
                  for (int q = 0; q < 8; ++q)
                      if (x[q] >= 0) a.cov[x[q]] = 1;
              }
          },
          [&](int u, int64_t b, int64_t e) {
              if (lane == 0) a.cov[u] = 1;
              if (u == s) return;
              if (lane == 0) te += (unsigned long long)(e - b);
              warp_row(a.col, b, e, lane, [&](int x) { a.cov[x] = 1; }, [] { return false; });
          });
}

template <typename Tm>
__device__ void run_p1(const P1Args &a, int ii, const Tm &tm, P1Smem &sm) {
    const Inst I = a.inst[ii];
    const int k = I.k, nv = I.nv, vb = (int)I.vbase;
    const int lane = threadIdx.x & 31;
    const int32_t *const hubs = a.hubs + a.hstart[ii];
    const int nh = (int)(a.hstart[ii + 1] - a.hstart[ii]);
    int32_t *const front[2] = {a.l_front0 + vb, a.l_front1 + vb};
    int32_t *const lsel = a.l_sel + vb;
    uint64_t *const rec[2] = {a.rec0 + vb, a.rec1 + vb};
    const int kbits = I.dbits + I.ibits;
    const int npass = (kbits + kDigitBits - 1) / kDigitBits > 0 ? (kbits + kDigitBits - 1) / kDigitBits : 1;
    const int top = npass * kDigitBits;
    const bool packed = kbits <= kOwnShift;
    const uint64_t idmask = (uint64_t(1) << I.ibits) - 1;
    auto part_of = [&](uint64_t r) { return packed ? (int)(r >> kOwnShift) : a.label[vb + (int)(r & idmask)]; };
    unsigned long long te = 0;

    if (threadIdx.x == 0) {
        sm.te = 0;
        sm.nfall = 0;
        sm.sh[0] = sm.sh[1] = P1Shared();
    }
    for (int p = threadIdx.x; p < kBatchMaxK; p += kP1Threads) {
        sm.psize[p] = 0;
        sm.npart[0][p] = sm.npart[1][p] = 0;
        sm.seeds[p] = -1;
    }
    for (int i = threadIdx.x; i < 2 * kBatchMaxK * kDigits; i += kP1Threads) (&sm.hist[0][0])[i] = 0;
    for (int i = tm.thread(); i < nv; i += tm.threads()) {
        a.label[vb + i] = -1;
        a.claim[vb + i] = INT_MAX;
        a.cov[vb + i] = 0;
    }
    tm.sync();
    int nseeds = 0, nfound = 0, rounds = 0;
    auto add_seed = [&](int v) {  // by every CTA alike
        if (threadIdx.x == 0) sm.seeds[nseeds] = v;
        ++nseeds;
        __syncthreads();
    };
    if (nv > 0) {
        // ---- seeds (seed.cpp:192-242) ----
        add_seed(vb + a.first[ii]);
        if (nh > 0)
            for (int p = 1, from = 0; p < k; ++p) {
                mark_ball(a, sm.seeds[nseeds - 1], tm, te);
                tm.sync();
                const int i = next_hub(a, hubs, nh, from, vb, nseeds, true, sm);
                if (i >= nh) break;
                add_seed(vb + hubs[i]);
                from = i + 1;
                tm.sync();  // every CTA has found the hub before its ball is marked
            }
        nfound = nseeds;
        // ---- seed completion (fewer than k seeds) ----
        for (int from = 0; nseeds < k;) {
            const int i = next_hub(a, hubs, nh, from, vb, nseeds, false, sm);
            if (i < nh) {
                add_seed(vb + hubs[i]);
                from = i + 1;
                continue;
            }
            from = nh;
            unsigned long long key = 0;
            for (int v = tm.thread(); v < nv; v += tm.threads()) {
                if (is_seed(sm, nseeds, vb + v)) continue;
                const unsigned long long c =
                    ((unsigned long long)(unsigned)deg_of(a, vb + v) << 32) | (0xffffffffull - (unsigned)v);
                key = c > key ? c : key;
            }
            key = team_max<kP1Threads>(key, tm, sm.wbest, &sm.cbest);
            if (key == 0) break;  // every vertex is a seed
            add_seed(vb + (int)(0xffffffffull - (key & 0xffffffffull)));
        }
        // ---- growth (partition.cpp:335-604) ----
        const int nstart = nseeds < k ? nseeds : k;
        if (tm.is_first())
            for (int p = threadIdx.x; p < nstart; p += kP1Threads) {
                const int s = sm.seeds[p];
                a.label[s] = p;
                front[0][p] = s;
                sm.psize[p] = 1;
                sm.npart[0][p] = 1;
            }
        tm.sync();
        int cur = 0, nfront = nstart, labelled = nstart;
        while (labelled < nv) {
            const int par = rounds & 1;
            P1Shared *const sh = tm.first(&sm.sh[par]);
            if (nfront == 0) {  // every frontier empty: all unlabelled vertices join the smallest part
                int bestp = 0;
                long long bs = 0;
                for (int p = 0; p < k; ++p) {
                    long long x = 0;
                    for (int r = 0; r < tm.size(); ++r) x += *tm.at(&sm.psize[p], r);
                    if (p == 0 || x < bs) {
                        bs = x;
                        bestp = p;
                    }
                }
                tm.sync();  // every CTA has read the sizes
                for (int i0 = tm.warp() * 32; i0 < nv; i0 += tm.threads()) {
                    const int v = vb + i0 + lane;
                    const bool un = i0 + lane < nv && a.label[v] < 0;
                    if (un) a.label[v] = bestp;
                    const int slot = warp_push(tm.first(&sm.nfall), un);
                    if (un) {
                        front[cur][slot] = v;
                        atomicAdd(&sm.npart[par][bestp], 1);
                    }
                }
                tm.sync();
                nfront = *tm.first(&sm.nfall);
                labelled += nfront;
                if (tm.is_first() && threadIdx.x == 0) sm.psize[bestp] += nfront;
            }
            // frontier vertices per part; need = min(count, theta)
            bool over = false;
            for (int p = threadIdx.x; p < k; p += kP1Threads) {
                int n = 0;
                for (int r = 0; r < tm.size(); ++r) n += *tm.at(&sm.npart[par][p], r);
                over = n > a.theta;
                sm.need[p] = n < a.theta ? n : a.theta;
            }
            over = __syncthreads_or(over);
            const int32_t *sel = front[cur];
            int nsel = nfront, ncarry = 0;
            int32_t *const nxtf = front[cur ^ 1];
            if (over) {
                // select need[p] smallest (degree, local id) per part: into lsel, the others carry over
                for (int i = tm.thread(); i < nfront; i += tm.threads()) {
                    const int v = front[cur][i], p = a.label[v];
                    const uint64_t key = ((uint64_t)deg_of(a, v) << I.ibits) | (uint64_t)(v - vb);
                    rec[0][i] = packed ? key | ((uint64_t)p << kOwnShift) : key;
                    atomicAdd(&sm.hist[0][p * kDigits + (int)((key >> (top - kDigitBits)) & (kDigits - 1))], 1);
                }
                tm.sync();
                int nlist = nfront;
                for (int pass = 0; pass < npass; ++pass) {
                    const int shift = top - kDigitBits * (pass + 1);
                    cut_digit(tm, k, sm.hist[pass & 1], sm.need, sm.below, sm.keep);
                    tm.sync();
                    const bool open = any_open(k, sm.keep);
                    for (int i = threadIdx.x; i < k * kDigits; i += kP1Threads) sm.hist[pass & 1][i] = 0;
                    const uint64_t *const list = rec[pass & 1];
                    uint64_t *const nxt = rec[(pass + 1) & 1];
                    for (int i0 = tm.warp() * 32; i0 < nlist; i0 += tm.threads()) {
                        const int i = i0 + lane;
                        bool take = false, keep = false, carry = false;
                        uint64_t r = 0;
                        int p = 0;
                        if (i < nlist) {
                            r = list[i];
                            p = part_of(r);
                            const int d = (int)((r >> shift) & (kDigits - 1));
                            take = d < sm.below[p];
                            keep = d == sm.keep[p];
                            carry = !take && !keep;
                        }
                        const int v = vb + (int)(r & idmask);
                        const int ts = warp_push(&sh->nsel, take);
                        if (take) lsel[ts] = v;
                        const int cs = warp_push(&sh->nnext, carry);
                        if (carry) {
                            nxtf[cs] = v;
                            atomicAdd(&sm.npart[par ^ 1][p], 1);
                        }
                        const int ks = warp_push(&sh->nact[pass], keep);
                        if (keep) {
                            nxt[ks] = r;
                            atomicAdd(&sm.hist[(pass + 1) & 1]
                                              [p * kDigits + (int)((r >> (shift - kDigitBits)) & (kDigits - 1))],
                                      1);
                        }
                    }
                    tm.sync();
                    if (!open) break;
                    nlist = sh->nact[pass];
                }
                sel = lsel;
                nsel = sh->nsel;
                ncarry = sh->nnext;
                tm.sync();  // every thread has read the carried count before claims are appended
            }
            // claims: atomicMin over part ids (partition.cpp:455-476); the first claim appends the vertex to
            // the next frontier
            visit(a.off, tm, nsel, [&](int i) { return sel[i]; },
                  [&](int, int64_t s, int64_t e) { return e - s > kP1Row; },
                  [&](bool act, int v, int64_t s, int64_t e) {
                      unsigned mine = 0;
                      if (act) {
                          const int p = a.label[v], n = (int)(e - s);
                          te += (unsigned long long)n;
                          for (int j = 0; j < n; j += 8) {
                              int u[8], l[8];
#pragma unroll
                              for (int q = 0; q < 8; ++q) u[q] = j + q < n ? __ldg(a.col + s + j + q) : -1;
#pragma unroll
                              for (int q = 0; q < 8; ++q) l[q] = u[q] >= 0 ? a.label[u[q]] : 0;
#pragma unroll
                              for (int q = 0; q < 8; ++q)
                                  if (l[q] < 0) l[q] = atomicMin(&a.claim[u[q]], p) == INT_MAX ? -1 : 0;
#pragma unroll
                              for (int q = 0; q < 8; ++q) mine |= l[q] < 0 ? 1u << (j + q) : 0u;
                          }
                      }
                      const int cnt = __popc(mine);
                      int incl = cnt;
                      for (int o = 1; o < 32; o <<= 1) {
                          const int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
                          if (lane >= o) incl += y;
                      }
                      int base = 0;
                      if (lane == 31 && incl) base = atomicAdd(&sh->nnext, incl);
                      int at = __shfl_sync(DMOLP_FULL_MASK, base, 31) + incl - cnt;
                      for (; mine; mine &= mine - 1) nxtf[at++] = __ldg(a.col + s + __ffs(mine) - 1);
                  },
                  [&](int v, int64_t s, int64_t e) {
                      const int p = a.label[v];
                      if (lane == 0) te += (unsigned long long)(e - s);
                      for (int64_t j0 = s; j0 < e; j0 += 128) {
                          int u[4];
                          bool f[4];
#pragma unroll
                          for (int q = 0; q < 4; ++q) u[q] = j0 + q * 32 + lane < e ? __ldg(a.col + j0 + q * 32 + lane) : -1;
#pragma unroll
                          for (int q = 0; q < 4; ++q) f[q] = u[q] >= 0 && a.label[u[q]] < 0;
#pragma unroll
                          for (int q = 0; q < 4; ++q)
                              if (f[q]) f[q] = atomicMin(&a.claim[u[q]], p) == INT_MAX;
                          unsigned m[4];
                          int tot = 0;
#pragma unroll
                          for (int q = 0; q < 4; ++q) {
                              m[q] = __ballot_sync(DMOLP_FULL_MASK, f[q]);
                              tot += __popc(m[q]);
                          }
                          if (tot == 0) continue;
                          int base = 0;
                          if (lane == 0) base = atomicAdd(&sh->nnext, tot);
                          base = __shfl_sync(DMOLP_FULL_MASK, base, 0);
#pragma unroll
                          for (int q = 0; q < 4; ++q) {
                              if (f[q]) nxtf[base + __popc(m[q] & ((1u << lane) - 1))] = u[q];
                              base += __popc(m[q]);
                          }
                      }
                  });
            tm.sync();
            // commit: claimed vertices take their part
            const int nnext = sh->nnext;
            for (int i = ncarry + tm.thread(); i < nnext; i += tm.threads()) {
                const int v = nxtf[i], p = a.claim[v];
                a.label[v] = p;
                a.claim[v] = INT_MAX;
                atomicAdd((unsigned long long *)&sm.psize[p], 1ull);
                atomicAdd(&sm.npart[par ^ 1][p], 1);
            }
            for (int p = threadIdx.x; p < k; p += kP1Threads) sm.npart[par][p] = 0;
            if (tm.is_first() && threadIdx.x == 0) sm.sh[par ^ 1] = P1Shared();
            tm.sync();
            labelled += nnext - ncarry;
            nfront = nnext;
            cur ^= 1;
            ++rounds;
        }
    }
    te = warp_sum_u64(te);
    if (lane == 0 && te) atomicAdd(tm.first(&sm.te), te);
    tm.sync();
    if (tm.is_first()) {
        if (threadIdx.x == 0) {
            P1Out o;
            o.nseeds_found = nfound;
            o.rounds = rounds;
            o.te = sm.te;
            a.out[ii] = o;
        }
        for (int p = threadIdx.x; p < kBatchMaxK; p += kP1Threads)
            a.seeds_out[(size_t)ii * kBatchMaxK + p] = p < k ? sm.seeds[p] : -1;
    }
    tm.sync();  // no CTA leaves, or starts on another graph, while its counters are read
}

__global__ void __launch_bounds__(kP1Threads, 2) k_batch_p1(P1Args a, const int32_t *order, int n) {
    __shared__ P1Smem sm;
    const CtaTeam<kP1Threads> tm;
    for (;;) {
        if (threadIdx.x == 0) sm.inst = atomicAdd(a.next, 1);
        __syncthreads();
        const int q = sm.inst;
        __syncthreads();
        if (q >= n) break;
        run_p1(a, order[q], tm, sm);
    }
}

__global__ void __launch_bounds__(kP1Threads, 2) k_batch_p1_team(P1Args a, const int32_t *order) {
    __shared__ P1Smem sm;
    const ClusterTeam<kP1Threads> tm;
    run_p1(a, order[blockIdx.x / tm.size()], tm, sm);
}

}  // namespace

int p1_threads() { return kP1Threads; }

int p1_max_team() {
    for (int c = kMaxTeam; c > 1; c >>= 1) {
        int n = 0;
        if (max_clusters(k_batch_p1_team, c, kP1Threads, &n) && n > 0) return c;
    }
    return 1;
}

void launch_p1(const P1Args &a, const int32_t *order, int grid, const TeamPlan &plan, const Fork &f, cudaStream_t s) {
    cudaMemsetAsync(a.next, 0, sizeof(int), s);
    f.open(plan, s);
    for (int j = 0, c = kMaxTeam; c > 1; ++j, c >>= 1) {
        if (plan.n[j] > 0) launch_cluster(k_batch_p1_team, plan.n[j], c, kP1Threads, f.stream(plan, j, s), a, order);
        order += plan.n[j];
    }
    const int n1 = plan.n[kTeamClasses - 1];
    if (n1 > 0) k_batch_p1<<<std::min(grid, n1), kP1Threads, 0, f.stream(plan, kTeamClasses - 1, s)>>>(a, order, n1);
    f.close(plan, s);
}

}  // namespace batch
}  // namespace dmolp
