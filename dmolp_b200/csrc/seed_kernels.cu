// Phase 1 on the resident CSR, in cooperative launches: the seeds, and the theta-limited multi-source BFS growth with
// all its rounds.
//
//   seeds   per seed, its radius-2 ball (compute_bfs with MAX_LEVELS = 3, src/phase1/seed.cpp:20-101) is OR-ed
//           into a coverage byte map: level 1 = the seed's row, level 2 = the rows of level 1; then the first
//           uncovered hub of maximum raw degree in hub order (seed.cpp:154-170) is the next seed: one 64-bit
//           atomicMax over (degree, ~hub_index).  A seed's ball covers it, so no hub is taken twice.
//   growth  rounds (partition.cpp:371-603): per part, the theta frontier vertices with the smallest (raw degree,
//           id) expand; an unlabelled neighbour is claimed by atomicMin over part ids, which is the reference's
//           "lowest part wins" (its parts are visited in ascending order with a shared visited set,
//           partition.cpp:455-476); claimed vertices join their part's frontier, unselected frontier vertices
//           carry over.
//
// What bounds it: latency.  A round handles at most theta vertices per part, a few dependent gathers each, and
// there are 20 to 80 rounds.  With a host check and seven launches per round a round cost 65 us on a 5 K-vertex
// mesh and 160 us on a skewed graph of a million vertices; here it is two grid barriers (claims | labels), a third
// when rows of more than kP1Piece arcs are split, and the select's only in rounds where a part has more than
// theta frontier vertices: 12 and 70 us a round.  Seeds and growth: 1.8 -> 0.5 ms on the mesh, 5.6 -> 2.2 ms on the
// skewed graph.
//
// Large graphs with few hubs get their hub list here, too (k_hub_stats, k_hub_top).
#include <algorithm>
#include <climits>

#include "select_radix.cuh"

namespace dmolp {
namespace {

constexpr int kP1Row = 16;     // rows of at most this many arcs are walked by one lane (a bit per claimed arc)
constexpr int kP1BlockV = 128;  // vertices per block of the launches: few blocks make a barrier cheap

// b.p1cnt: frontier sizes and queued row pieces by round parity, labelled vertices, rounds, seeds found
enum { kFront = 0, kPieces = 2, kLabelled = 4, kRounds = 5, kFound = 6 };

// The first warp of every block comes first, so short lists spread over the SMs.
__device__ __forceinline__ int grid_warp() { return (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x; }
__device__ __forceinline__ int grid_warps() { return (int)(blockDim.x >> 5) * (int)gridDim.x; }

// Row [s, e) of vertex v queued in pieces of kP1Piece arcs.  The queue's narcs / 256 + 2 places are enough for every row
// once (at least kP1Piece / 2 arcs a piece), so between two resets of the counter no row is queued twice.
__device__ __forceinline__ void queue_row(const Buffers &b, int *ctr, int v, int64_t deg) {
    const int n = (int)((deg + kP1Piece - 1) / kP1Piece);
    const int q = atomicAdd(ctr, n);
    for (int i = 0; i < n; ++i) b.chunkq[q + i] = make_int2(v, i * kP1Piece);
}

__device__ __forceinline__ void cover_arcs(const Buffers &b, int64_t s, int64_t e) {
    warp_row(b.col, s, e, threadIdx.x & 31, [&](int x) { b.covered[x] = 1; }, [] { return false; });
}

// seeds[0, found) to b.need, found to p1cnt.  b.covered, b.best[2] and p1cnt are zero on entry.  repeats: rows may list
// an id more than once (b.claim is then zero on entry); the first occurrence of a neighbour in the seed's row claims
// its place in the queue, the others only count its arcs, as a walk of each occurrence would.
__global__ void __launch_bounds__(kSelThreads, 1) k_p1_find_seeds(Buffers b, int k, int first, int nhubs, int repeats,
                                                                  unsigned int polls) {
    const int lane = threadIdx.x & 31;
    int seed = first, found = 1;
    unsigned long long te = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) b.need[0] = first;
    for (int p = 1; p < k; ++p) {
        int *const npiece = &b.p1cnt[kPieces + (p & 1)];
        const int64_t s = b.off[seed], e = b.off[seed + 1];
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            b.covered[seed] = 1;
            te += (unsigned long long)(e - s);
        }
        for (int64_t i0 = s + (int64_t)grid_warp() * 32; i0 < e; i0 += (int64_t)grid_warps() * 32) {
            const int64_t i = i0 + lane;
            int64_t us = 0, ue = 0;
            if (i < e) {
                const int u = b.col[i];
                b.covered[u] = 1;
                if (u != seed) {
                    us = b.off[u];
                    ue = b.off[u + 1];
                    te += (unsigned long long)(ue - us);
                    if (ue - us > kP1Piece && (!repeats || atomicExch(&b.claim[u], p) != p))
                        queue_row(b, npiece, u, ue - us);
                }
            }
            const int64_t deg = ue - us;
            if (deg <= kP1Row)
                for (int64_t j = us; j < ue; j += 8) {
                    int x[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) x[q] = j + q < ue ? __ldg(b.col + j + q) : -1;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (x[q] >= 0) b.covered[x[q]] = 1;
                }
            for (unsigned m = __ballot_sync(DMOLP_FULL_MASK, deg > kP1Row && deg <= kP1Piece); m; m &= m - 1) {
                const int l = __ffs(m) - 1;
                cover_arcs(b, __shfl_sync(DMOLP_FULL_MASK, us, l), __shfl_sync(DMOLP_FULL_MASK, ue, l));
            }
        }
        if (!grid_sync(b.ctrl, polls, 20)) return;
        const int np = __ldcg(npiece);
        if (np) {  // the same in every block
            for (int q = grid_warp(); q < np; q += grid_warps()) {
                const int2 c = b.chunkq[q];
                const int64_t ps = b.off[c.x] + c.y, pe = b.off[c.x + 1];
                cover_arcs(b, ps, pe - ps > kP1Piece ? ps + kP1Piece : pe);
            }
            if (!grid_sync(b.ctrl, polls, 21)) return;
        }
        // the next seed; the other parity's maximum and piece count were last read before the barrier above
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            b.best[(p + 1) & 1] = 0;
            b.p1cnt[kPieces + ((p + 1) & 1)] = 0;
        }
        unsigned long long best = 0;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nhubs; i += gridDim.x * blockDim.x) {
            const int h = b.hubs[i];
            if (b.covered[h]) continue;
            const unsigned long long key = ((unsigned long long)(unsigned)b.rawdeg[h] << 32) |
                                           (unsigned long long)(0xffffffffu - (unsigned)i);
            best = best > key ? best : key;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ob = __shfl_xor_sync(DMOLP_FULL_MASK, best, o);
            best = best > ob ? best : ob;
        }
        if (lane == 0 && best) atomicMax(&b.best[p & 1], best);
        if (!grid_sync(b.ctrl, polls, 22)) return;
        best = __ldcg(&b.best[p & 1]);
        if (best == 0) break;  // the same in every block
        seed = b.hubs[0xffffffffu - (unsigned)(best & 0xffffffffull)];
        if (blockIdx.x == 0 && threadIdx.x == 0) b.need[p] = seed;
        ++found;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) b.p1cnt[kFound] = found;
    te = warp_sum_u64(te);
    if (lane == 0 && te) atomicAdd(b.p1te, te);
}

// A warp's appends to the next frontier, collected in shared memory: the counter is one address, and with an append
// per step and warp the 25 K row pieces of one round of a skewed graph of a million vertices took 90 us, not 61.
constexpr int kStageP1 = 512;
struct Append {
    int32_t *stage, *next;
    int *nnext;
    int n;  // staged, the same in every lane
    __device__ __forceinline__ void flush() {
        const int lane = threadIdx.x & 31;
        int base = 0;
        if (lane == 0 && n) base = atomicAdd(nnext, n);
        base = __shfl_sync(DMOLP_FULL_MASK, base, 0);
        __syncwarp();
        for (int i = lane; i < n; i += 32) next[base + i] = stage[i];
        __syncwarp();
        n = 0;
    }
    // Room for cnt entries of this lane; all lanes call it, and fewer than kStageP1 are asked for together.
    __device__ __forceinline__ int32_t *take(int cnt) {
        const int lane = threadIdx.x & 31;
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
            if (lane >= o) incl += y;
        }
        const int tot = __shfl_sync(DMOLP_FULL_MASK, incl, 31);
        if (n + tot > kStageP1) flush();
        int32_t *const r = stage + n + incl - cnt;
        n += tot;
        return r;
    }
};

// Claims of the arcs [s, e) of frontier vertices by one warp: unlabelled neighbours take atomicMin(part), and the one
// thread that turns a claim from INT_MAX appends the vertex to the next frontier, as ~vertex.  All lanes call it;
// the G lanes of a group hold the same row (s == e: none), part p, and walk it G * U arcs a step, so that a warp has
// 32 / G rows in flight.
template <int G, int U>
__device__ __forceinline__ void claim_rows(const Buffers &b, int p, int64_t s, int64_t e, Append &out) {
    for (int64_t j0 = s + (threadIdx.x & (G - 1)); __any_sync(DMOLP_FULL_MASK, j0 < e); j0 += G * U) {
        int u[U];
        bool f[U];
        int cnt = 0;
#pragma unroll
        for (int q = 0; q < U; ++q) u[q] = j0 + q * G < e ? __ldg(b.col + j0 + q * G) : -1;
#pragma unroll
        for (int q = 0; q < U; ++q) f[q] = u[q] >= 0 && b.label[u[q]] < 0;
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (f[q]) {
                f[q] = atomicMin(&b.claim[u[q]], p) == INT_MAX;
                cnt += f[q];
            }
        if (!__any_sync(DMOLP_FULL_MASK, cnt > 0)) continue;
        int32_t *slot = out.take(cnt);
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (f[q]) *slot++ = ~u[q];
    }
}

// All rounds from the seeds b.need[0, k) (-1: the part has none).  npart2[2]: frontier vertices per part, by round
// parity.  smem_off: words of dynamic shared memory in front of this kernel's own 2k counters (the select's,
// then the warps' staged appends).
__global__ void __launch_bounds__(kSelThreads, 1) k_p1_grow(Buffers b, const SelArgs a, int nv, int k, int theta, int ibits,
                                                            int smem_off) {
    extern __shared__ unsigned int smem[];
    int *const s_np = reinterpret_cast<int *>(smem) + smem_off;  // frontier vertices per part, next round
    int *const s_ps = s_np + k;                                  // vertices labelled per part
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int32_t *const npart2[2] = {b.npart, b.sel_below};
    LpControl *const ctl = a.ctl;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        b.label[v] = -1;
        b.claim[v] = INT_MAX;
    }
    if (blockIdx.x == 0) {
        for (int p = threadIdx.x; p < k; p += blockDim.x) {
            const int has = b.need[p] >= 0;
            b.psize[p] = has;
            npart2[0][p] = has;
            npart2[1][p] = 0;
        }
        if (threadIdx.x < 8) b.p1cnt[threadIdx.x] = 0;
    }
    if (!grid_sync(ctl, a.polls, 23)) return;
    if (blockIdx.x == 0)
        for (int p = threadIdx.x; p < k; p += blockDim.x) {
            const int s = b.need[p];
            if (s < 0) continue;
            b.label[s] = p;
            b.win[0][atomicAdd(&b.p1cnt[kFront], 1)] = s;
            atomicAdd(&b.p1cnt[kLabelled], 1);
        }
    if (!grid_sync(ctl, a.polls, 24)) return;
    unsigned long long te = 0;
    int rounds = 0;
    for (int par = 0; __ldcg(&b.p1cnt[kLabelled]) < nv; par ^= 1, ++rounds) {
        int32_t *const front = b.win[par], *const next = b.win[par ^ 1];
        int *const nnext = &b.p1cnt[kFront + (par ^ 1)], *const npiece = &b.p1cnt[kPieces + par];
        int n = __ldcg(&b.p1cnt[kFront + par]);
        for (int p = threadIdx.x; p < 2 * k; p += blockDim.x) s_np[p] = 0;
        if (n == 0) {
            // every frontier empty (partition.cpp:376-394): the unlabelled vertices join the smallest part
            int best = 0;
            long long bs = __ldcg(b.psize);
            for (int p = 1; p < k; ++p) {
                const long long x = __ldcg(b.psize + p);
                if (x < bs) {
                    bs = x;
                    best = p;
                }
            }
            if (!grid_sync(ctl, a.polls, 25)) return;  // every block has read the sizes
            for (int v0 = grid_warp() * 32; v0 < nv; v0 += grid_warps() * 32) {
                const int v = v0 + lane;
                const bool un = v < nv && b.label[v] < 0;
                if (un) b.label[v] = best;
                const unsigned m = __ballot_sync(DMOLP_FULL_MASK, un);
                int base = 0;
                if (lane == 0 && m) {
                    base = atomicAdd(&b.p1cnt[kFront + par], __popc(m));
                    atomicAdd(&s_ps[0], __popc(m));  // (any slot: only the sum is used here)
                }
                base = __shfl_sync(DMOLP_FULL_MASK, base, 0);
                if (un) front[base + __popc(m & ((1u << lane) - 1))] = v;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                const int c = s_ps[0];
                s_ps[0] = 0;
                if (c) {
                    atomicAdd(&b.p1cnt[kLabelled], c);
                    atomicAdd(&npart2[par][best], c);
                    atomicAdd((unsigned long long *)&b.psize[best], (unsigned long long)c);
                }
            }
            if (!grid_sync(ctl, a.polls, 26)) return;
            n = __ldcg(&b.p1cnt[kFront + par]);
        }
        bool over = false;
        for (int p = threadIdx.x; p < k; p += blockDim.x) over |= __ldcg(npart2[par] + p) > theta;
        over = __syncthreads_or(over);  // (and the cleared counters, and the last round's staged appends are out)
        const int cap = (n + (int)gridDim.x - 1) / (int)gridDim.x;
        const int lo = (int)blockIdx.x * cap, hi = min(n, lo + cap);  // this block's frontier slots
        if (over) {
            for (int i = lo + (int)threadIdx.x; i < hi; i += blockDim.x) {
                const int v = front[i];
                b.bown[i] = b.label[v];
                b.bkey[i] = ((uint64_t)(unsigned)b.rawdeg[v] << ibits) | (uint64_t)v;
                b.bsel[i] = 0;
            }
            __syncthreads();
            const int how = select_body<false>(a, n, npart2[par]);
            if (how == 0) return;
            if (how == 2 && !grid_sync(ctl, a.polls, 27)) return;  // block 0 marked other blocks' records
        }
        // ---- claims of the selected vertices' arcs; the others carry over.  Few rows: eight lanes each; else a
        //      lane per row of at most kP1Row arcs, eight lanes per longer one ----
        Append out = {reinterpret_cast<int32_t *>(smem) + wib * kStageP1, next, nnext, 0};  // (the select is done)
        const bool few = cap <= (int)(blockDim.x >> 3);  // the same in every block
        const int step = few ? (int)(blockDim.x >> 3) : (int)blockDim.x;
        for (int i0 = lo + (few ? wib * 4 : wib * 32); i0 < hi; i0 += step) {
            const int i = i0 + (few ? lane >> 3 : lane);
            const bool lead = !few || (lane & 7) == 0;
            int v = 0, p = 0, mine = 0;  // a bit per arc whose neighbour this lane claimed first
            int64_t s = 0, e = 0;
            bool carry = false;
            if (i < hi) {
                v = front[i];
                p = b.label[v];
                if (!over || b.bsel[i]) {
                    s = b.off[v];
                    e = b.off[v + 1];
                    if (lead) te += (unsigned long long)(e - s);
                    if (e - s > kP1Piece) {
                        if (lead) queue_row(b, npiece, v, e - s);
                        e = s;
                    }
                } else if (lead) {
                    carry = true;
                    atomicAdd(&s_np[p], 1);
                }
            }
            const int deg = (int)(e - s);
            if (!few && deg <= kP1Row)
                for (int j = 0; j < deg; j += 8) {
                    int u[8];
                    bool f[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) u[q] = j + q < deg ? __ldg(b.col + s + j + q) : -1;
#pragma unroll
                    for (int q = 0; q < 8; ++q) f[q] = u[q] >= 0 && b.label[u[q]] < 0;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (f[q] && atomicMin(&b.claim[u[q]], p) == INT_MAX) mine |= 1 << (j + q);
                }
            const int cnt = carry ? 1 : __popc(mine);
            if (__any_sync(DMOLP_FULL_MASK, cnt > 0)) {
                int32_t *slot = out.take(cnt);
                if (carry) *slot = v;
                for (unsigned m = (unsigned)mine; m; m &= m - 1) *slot++ = ~__ldg(b.col + s + __ffs(m) - 1);
            }
            if (few) {
                claim_rows<8, 4>(b, p, s, e, out);
            } else {
                for (unsigned m = __ballot_sync(DMOLP_FULL_MASK, deg > kP1Row); m;) {
                    int l = 32;  // the group's row: the (lane / 8)-th of the next four
                    for (int g = 0; g < 4; ++g) {
                        if (g == (lane >> 3) && m) l = __ffs(m) - 1;
                        m &= m - 1;
                    }
                    const int src = l & 31;
                    const int pl = __shfl_sync(DMOLP_FULL_MASK, p, src);
                    const int64_t sl = __shfl_sync(DMOLP_FULL_MASK, s, src), el = __shfl_sync(DMOLP_FULL_MASK, e, src);
                    claim_rows<8, 8>(b, pl, sl, l < 32 ? el : sl, out);
                }
            }
        }
        out.flush();
        if (!grid_sync(ctl, a.polls, 28)) return;
        const int np = __ldcg(npiece);
        if (np) {  // the same in every block
            for (int q = grid_warp(); q < np; q += grid_warps()) {
                const int2 c = b.chunkq[q];
                const int64_t ps = b.off[c.x] + c.y, pe = b.off[c.x + 1];
                claim_rows<32, 4>(b, b.label[c.x], ps, pe - ps > kP1Piece ? ps + kP1Piece : pe, out);
            }
            out.flush();
            if (!grid_sync(ctl, a.polls, 29)) return;
        }
        // ---- claimed vertices take their part ----
        const int nn = __ldcg(nnext);
        for (int i = grid_warp() * 32 + lane; i < nn; i += grid_warps() * 32) {
            const int v = ~next[i];
            if (v < 0) continue;  // carried over
            next[i] = v;
            const int p = __ldcg(b.claim + v);
            b.label[v] = p;
            atomicAdd(&s_np[p], 1);
            atomicAdd(&s_ps[p], 1);
        }
        __syncthreads();
        int labelled = 0;
        for (int p = threadIdx.x; p < k; p += blockDim.x) {
            if (s_np[p]) atomicAdd(&npart2[par ^ 1][p], s_np[p]);
            if (s_ps[p]) atomicAdd((unsigned long long *)&b.psize[p], (unsigned long long)s_ps[p]);
            labelled += s_ps[p];
        }
        for (int o = 16; o > 0; o >>= 1) labelled += __shfl_xor_sync(DMOLP_FULL_MASK, labelled, o);
        if (lane == 0 && labelled) atomicAdd(&b.p1cnt[kLabelled], labelled);
        if (blockIdx.x == 0) {  // this round's frontier and the other parity's pieces were read before the last barrier
            for (int p = threadIdx.x; p < k; p += blockDim.x) npart2[par][p] = 0;
            if (threadIdx.x == 0) {
                b.p1cnt[kFront + par] = 0;
                b.p1cnt[kPieces + (par ^ 1)] = 0;
            }
        }
        if (!grid_sync(ctl, a.polls, 30)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) b.p1cnt[kRounds] = rounds;
    te = warp_sum_u64(te);
    if (lane == 0 && te) atomicAdd(b.p1te, te);
}

// ------------------------------------------------------------------------------------ hub list
// Degree statistics: total, maximum D, then find_first_seed's closed form (hubsort.cpp, first_seed_of).
__global__ void __launch_bounds__(kSelThreads, 1) k_hub_stats(Buffers b, LpControl *ctl, int nv, unsigned int polls) {
    HubState *const h = b.hubst;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        h->total = 0;
        h->dmax = INT_MIN;
        h->vhigh = -1;
        h->vlow = INT_MAX;
    }
    if (!grid_sync(ctl, polls, 50)) return;
    unsigned long long sum = 0;
    int mx = INT_MIN;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        const int d = b.rawdeg[v];
        sum += (unsigned long long)d;
        mx = max(mx, d);
    }
    sum = warp_sum_u64(sum);
    mx = __reduce_max_sync(DMOLP_FULL_MASK, mx);
    if ((threadIdx.x & 31) == 0) {
        if (sum) atomicAdd(&h->total, sum);
        atomicMax(&h->dmax, mx);
    }
    if (!grid_sync(ctl, polls, 51)) return;
    const int D = __ldcg(&h->dmax);
    int hi = -1, lo = INT_MAX;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x)
        if (b.rawdeg[v] == D) {
            hi = max(hi, v);
            if (v < D) lo = min(lo, v);
        }
    if (hi >= 0) atomicMax(&h->vhigh, hi);
    if (lo != INT_MAX) atomicMin(&h->vlow, lo);
}

// The swap of libstdc++'s median-of-three: the pivot to position r.
__device__ __forceinline__ void median_swap(int2 *a, int r, int x, int y, int z) {
    const int dx = a[x].y, dy = a[y].y, dz = a[z].y;
    int m;
    if (dx < dy) m = dy < dz ? y : (dx < dz ? z : x);
    else m = dx < dz ? x : (dy < dz ? z : y);
    const int2 t = a[r];
    a[r] = a[m];
    a[m] = t;
}

// std::sort's partitions of (vertex, degree) pairs by degree, followed into the right side while it holds position t0
// (hubsort.cpp, top_by_degree, does the same on the host: 1.9 ms for a million pairs; the whole list now takes 0.21).
// Hoare's scans pair the k-th position from the left whose degree is not below the pivot's with the k-th from the right
// whose degree is not above it, and swap while the left one lies before the right one.  With l(p) such positions left
// of p and r(p) at or right of it, the number of swaps is the maximum over p of min(l(p), r(p)); l grows and r falls,
// so the maximum lies in the block's slice where they cross.  The cut is the next left position, or the last swapped
// right one if that comes first.  Per partition: pivot | counts | pairs listed by rank | swaps, a barrier each.
__global__ void __launch_bounds__(kSelThreads, 1) k_hub_top(Buffers b, LpControl *ctl, int nv, int t0, int depth,
                                                            unsigned int polls) {
    constexpr int kW = kSelThreads / 32, kMaxGrid = 256;
    __shared__ int s_l[kW], s_r[kW], s_bl[kMaxGrid + 1], s_br[kMaxGrid + 1], s_star, s_m;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = gridDim.x, B = blockIdx.x;
    const unsigned upto = lane == 31 ? ~0u : (2u << lane) - 1u;  // this lane and those below
    int2 *const a = reinterpret_cast<int2 *>(b.dlkey);
    int *const blk = reinterpret_cast<int *>(b.psize);  // [2 * G] counts of every block
    int32_t *const posl = b.cand, *const posr = b.bv;
    HubState *const h = b.hubst;
    for (int i = B * blockDim.x + threadIdx.x; i < nv; i += G * blockDim.x)
        a[i] = make_int2(nv - 1 - i, b.rawdeg[nv - 1 - i]);
    if (B == 0 && threadIdx.x == 0) h->cutl[0] = h->cutl[1] = INT_MAX;
    if (!grid_sync(ctl, polls, 52)) return;
    int first = 0, split = -1;
    for (int par = 0; nv - first > kHubHostMax && depth > 0; par ^= 1) {
        --depth;
        if (B == 0 && threadIdx.x == 0) {
            median_swap(a, first, first + 1, first + (nv - first) / 2, nv - 1);
            h->cutl[par ^ 1] = INT_MAX;  // last read before the last barrier
        }
        if (!grid_sync(ctl, polls, 53)) return;
        const int pv = a[first].y, lo0 = first + 1, n = nv - lo0;
        const int len = (n + G - 1) / G, wlen = ((len + kW - 1) / kW + 31) & ~31;
        // warp w's share [x, y) of block sb's slice
        auto share = [&](int sb, int &x, int &y) {
            const int s = lo0 + min(n, sb * len), e = lo0 + min(n, (sb + 1) * len);
            x = min(e, s + w * wlen);
            y = min(e, x + wlen);
        };
        auto count = [&](int sb) {
            int x, y, cl = 0, cr = 0;
            share(sb, x, y);
            for (int i = x + lane; i < y; i += 32) {
                const int d = a[i].y;
                cl += d >= pv;
                cr += d <= pv;
            }
            cl = __reduce_add_sync(DMOLP_FULL_MASK, cl);
            cr = __reduce_add_sync(DMOLP_FULL_MASK, cr);
            if (lane == 0) {
                s_l[w] = cl;
                s_r[w] = cr;
            }
            __syncthreads();
        };
        // counts in front of warp w's share, from the slice's start
        auto before = [&](int &cl, int &cr) {
            cl = __reduce_add_sync(DMOLP_FULL_MASK, lane < w ? s_l[lane] : 0);
            cr = __reduce_add_sync(DMOLP_FULL_MASK, lane < w ? s_r[lane] : 0);
        };
        count(B);
        if (w == 0) {
            const int cl = __reduce_add_sync(DMOLP_FULL_MASK, s_l[lane]), cr = __reduce_add_sync(DMOLP_FULL_MASK, s_r[lane]);
            if (lane == 0) {
                blk[B] = cl;
                blk[G + B] = cr;
            }
        }
        int myl, myr;
        before(myl, myr);
        if (!grid_sync(ctl, polls, 54)) return;
        if (w == 0) {  // exclusive prefixes over the blocks
            int bl = 0, br = 0;
            for (int j0 = 0; j0 < G; j0 += 32) {
                const int j = j0 + lane;
                const int cl = j < G ? __ldcg(blk + j) : 0, cr = j < G ? __ldcg(blk + G + j) : 0;
                int il = cl, ir = cr;
                for (int o = 1; o < 32; o <<= 1) {
                    const int yl = __shfl_up_sync(DMOLP_FULL_MASK, il, o), yr = __shfl_up_sync(DMOLP_FULL_MASK, ir, o);
                    if (lane >= o) {
                        il += yl;
                        ir += yr;
                    }
                }
                if (j < G) {
                    s_bl[j + 1] = bl + il;
                    s_br[j + 1] = br + ir;
                }
                bl += __shfl_sync(DMOLP_FULL_MASK, il, 31);
                br += __shfl_sync(DMOLP_FULL_MASK, ir, 31);
            }
            if (lane == 0) {
                s_bl[0] = s_br[0] = 0;
                s_star = INT_MAX;
            }
        }
        __syncthreads();
        const int totr = s_br[G];
        for (int j = threadIdx.x; j < G; j += blockDim.x)
            if (s_bl[j + 1] >= totr - s_br[j + 1]) atomicMin(&s_star, j);
        __syncthreads();
        const int star = s_star;  // the slice in which the counts cross (the last slice: r is 0 at its end)
        if (threadIdx.x == 0) s_m = min(s_bl[star], totr - s_br[star]);
        count(star);
        {
            int x, y, cl, cr, best = 0;
            before(cl, cr);
            cl += s_bl[star];
            cr += s_br[star];
            share(star, x, y);
            for (int i0 = x; i0 < y; i0 += 32) {
                const int i = i0 + lane;
                const int d = i < y ? a[i].y : 0;
                const unsigned ml = __ballot_sync(DMOLP_FULL_MASK, i < y && d >= pv);
                const unsigned mr = __ballot_sync(DMOLP_FULL_MASK, i < y && d <= pv);
                if (i < y) best = max(best, min(cl + __popc(ml & upto), totr - cr - __popc(mr & upto)));
                cl += __popc(ml);
                cr += __popc(mr);
            }
            best = __reduce_max_sync(DMOLP_FULL_MASK, best);
            if (lane == 0) atomicMax(&s_m, best);
        }
        __syncthreads();
        const int m = s_m;  // swaps; the same in every block
        {
            int x, y, cl = s_bl[B] + myl, cr = s_br[B] + myr;
            share(B, x, y);
            for (int i0 = x; i0 < y; i0 += 32) {
                const int i = i0 + lane;
                const int d = i < y ? a[i].y : 0;
                const bool left = i < y && d >= pv, right = i < y && d <= pv;
                const unsigned ml = __ballot_sync(DMOLP_FULL_MASK, left), mr = __ballot_sync(DMOLP_FULL_MASK, right);
                const int rl = cl + __popc(ml & upto) - 1;         // 0-based from the left
                const int rr = totr - (cr + __popc(mr & upto));    // 0-based from the right
                if (left && rl < m) posl[rl] = i;
                if (left && rl == m) h->cutl[par] = i;
                if (right && rr < m) posr[rr] = i;
                cl += __popc(ml);
                cr += __popc(mr);
            }
        }
        if (!grid_sync(ctl, polls, 55)) return;
        const int cut = min(__ldcg(&h->cutl[par]), m > 0 ? __ldcg(posr + m - 1) : INT_MAX);
        for (int q = B * blockDim.x + threadIdx.x; q < m; q += G * blockDim.x) {
            const int i = posl[q], j = posr[q];
            const int2 t = a[i];
            a[i] = a[j];
            a[j] = t;
        }
        if (!grid_sync(ctl, polls, 56)) return;
        if (cut > t0) {
            split = cut;
            break;
        }
        first = cut;
    }
    if (B == 0 && threadIdx.x == 0) {
        h->first = first;
        h->depth = depth;
        h->cut = split;
    }
}

size_t grow_smem(int k, int *off) {
    const size_t stage = (size_t)(kSelThreads / 32) * kStageP1 * sizeof(int32_t);
    const size_t sel = std::max((select_smem_bytes(k) + 15) & ~(size_t)15, stage);
    if (off) *off = (int)(sel / sizeof(int));
    return sel + 2 * (size_t)k * sizeof(int);
}

// All blocks are resident: at most one per SM, a cooperative launch.
template <typename K, typename... A>
void launch_resident(dmolp_ctx *c, K kernel, size_t smem, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min<int64_t>(c->num_sms, std::max<int64_t>(8, (c->nv + kP1BlockV - 1) / kP1BlockV)));
    cfg.blockDim = dim3(kSelThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess && c->launch_error == cudaSuccess) c->launch_error = e;  // reported by the entry point
    c->launches += 1;
}

}  // namespace

void p1_hub_stats(dmolp_ctx *c) {
    launch_resident(c, k_hub_stats, 0, c->b, c->b.ctrl, (int)c->nv, c->wait_polls);
}

void p1_hub_top(dmolp_ctx *c, int64_t t0, int depth) {
    launch_resident(c, k_hub_top, 0, c->b, c->b.ctrl, (int)c->nv, (int)t0, depth, c->wait_polls);
}

void p1_find_seeds(dmolp_ctx *c, int k, int first, int64_t nhubs) {
    launch_resident(c, k_p1_find_seeds, 0, c->b, k, first, (int)nhubs, c->rows_sorted ? 0 : 1, c->wait_polls);
}

void p1_grow(dmolp_ctx *c, int k, int theta) {
    int off = 0;
    const size_t smem = grow_smem(k, &off);
    SelArgs a = select_args(c, k, c->rbits + c->ibits);
    a.theta = theta;
    launch_resident(c, k_p1_grow, smem, c->b, a, (int)c->nv, k, theta, c->ibits, off);
}

void p1_prepare() {
    size_t m = 0;
    for (int k : {kSmemSegMax, (int)DMOLP_MAX_K}) m = std::max(m, grow_smem(k, nullptr));
    cudaFuncSetAttribute(k_p1_grow, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)m);
}

}  // namespace dmolp
