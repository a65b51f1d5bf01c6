// Input features of the learned proposal, computed on the device for every graph of a batch:
//
//   anchors  eight vertices per graph by farthest-point sampling over hop distance (the first: the lowest id
//            of maximum degree).  A team of CTAs per graph (team.cuh) runs all eight searches in one launch,
//            a barrier of the team per level.  From the second anchor on a search visits only the vertices
//            that are closer to it than to every earlier anchor: the running minimum changes nowhere else
//            (it is 1-Lipschitz along arcs), and the search ends as soon as its cell is full.
//   walk     lazy random walks from the anchors, eight channels per vertex: P' = P/2 + (sum over neighbours
//            of P/deg)/2, T steps (the first anchor's eccentricity, at most 96), float32 sums in row order.
//   features log landing probabilities standardised per graph, degree / mean degree, log(1 + degree), k / 64.
//
// What bounds it: the searches by latency (a level of a mesh is a handful of vertices, about five dependent L2
// accesses and a barrier); the walk by L2, 36 bytes per arc and step.  Before, a level was a launch over all
// graphs (64 mixed graphs took 2752 of them, 24 ms; now about 5 ms), and a skewed graph walked its hub rows with
// one thread (7.7 ms a step at a million vertices; now 0.64 ms).  The walk's chunks stay at about 120 us a step
// for 1.3 M walking vertices: 32-byte gathers at 3.9 TB/s.  Tried on them without gain: four lanes of two channels
// (8.8 instead of 7.3 ms for the skewed graph's features), groups of graphs whose state stays in L2 (one launch
// per group and step: 21.9 instead of 18.8 ms).
//
// Work units of the walk and of the per-vertex passes are chunks of at most kChunkV consecutive vertices of one
// graph, ordered by their graph's steps, so that a step launches exactly the chunks that still walk.
#include <algorithm>
#include <climits>
#include <numeric>
#include <vector>

#include "lp_device.cuh"
#include "mpnn.cuh"
#include "team.cuh"

namespace dmolp {
namespace mpnn {
namespace {

using batch::ClusterTeam;
using batch::CtaTeam;
using batch::GridTeam;
using batch::Inst;

constexpr int kAncThreads = 512;
constexpr int kAncRow = 32;     // rows of at most this many arcs are searched by two lanes
constexpr int kHugeRow = 4096;  // longer rows are searched by the whole team
// A graph whose share of the batch is more than this many CTAs gets that share as a team of a cooperative launch: from
// twice a cluster's 16 on, more CTAs beat the cheaper barrier (features of a skewed graph alone, 1 M vertices: 6.5 -> 4.6 ms).
constexpr int kGridShare = 32;
constexpr int kGridTeams = 4;  // at most 148 / 32
constexpr int kWalkU = 16;      // walk: arcs in flight per vertex
using batch::kLongRow;          // walk: longer rows are summed by a block of their own

// A vertex's row and state in one 16-byte load.
__device__ __forceinline__ SearchRow load_row(const SearchRow *p) {
    const int4 x = *reinterpret_cast<const int4 *>(p);
    SearchRow r;
    r.start = (int64_t)(((uint64_t)(unsigned)x.y << 32) | (unsigned)x.x);
    r.len = x.z;
    r.dist = x.w;
    return r;
}

// What the team shares: in the first CTA's shared memory, or (GridTeam) in global memory.
struct AncShared {
    int cnt[3];   // frontier counts, rotating: level L reads cnt[L % 3], fills the next, clears the one after
    int nhuge[2];
    unsigned int word;                  // GridTeam: its barrier,
    unsigned long long best[kAnchors];  // and the maxima of the anchors' keys; zero before the launch
};

struct AncSmem {
    unsigned long long wbest[kAncThreads / 32], cbest;
    AncShared sh;
    int inst;
};

// The team's maximum of a key, for anchor j.
template <typename Tm>
__device__ __forceinline__ bool anchor_max(unsigned long long &key, int, const Tm &tm, AncSmem &sm, AncShared &) {
    key = batch::team_max<kAncThreads>(key, tm, sm.wbest, &sm.cbest);
    return true;
}
__device__ __forceinline__ bool anchor_max(unsigned long long &key, int j, const GridTeam<kAncThreads> &tm, AncSmem &,
                                           AncShared &sh) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(DMOLP_FULL_MASK, key, o);
        key = y > key ? y : key;
    }
    if ((threadIdx.x & 31) == 0 && key) atomicMax(&sh.best[j], key);
    if (!tm.sync()) return false;
    key = __ldcg(&sh.best[j]);
    return true;
}

// Arcs [s, e) searched by a warp: neighbours farther than d get d and join list.
__device__ __forceinline__ void search_arcs(const FeatWork &w, int64_t s, int64_t e, int d, int *ctr, SearchRow *list) {
    const int lane = threadIdx.x & 31;
    for (int64_t j0 = s; j0 < e; j0 += 128) {
        int u[4];
        SearchRow x[4];
        bool f[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) u[q] = j0 + q * 32 + lane < e ? __ldg(w.col + j0 + q * 32 + lane) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[q].dist = 0;
            if (u[q] >= 0) x[q] = load_row(w.row + u[q]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) f[q] = x[q].dist > d && atomicMin(&w.row[u[q]].dist, d) > d;
        unsigned m[4];
        int tot = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            m[q] = __ballot_sync(DMOLP_FULL_MASK, f[q]);
            tot += __popc(m[q]);
        }
        if (tot == 0) continue;
        int base = 0;
        if (lane == 0) base = atomicAdd(ctr, tot);
        base = __shfl_sync(DMOLP_FULL_MASK, base, 0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (f[q]) list[base + __popc(m[q] & ((1u << lane) - 1))] = x[q];
            base += __popc(m[q]);
        }
    }
}

// One level: the neighbours of the nf frontier rows that are farther than L + 1 form the next frontier, at
// distance L + 1.  Two lanes per row of at most kAncRow arcs, eight arcs each in flight, so that a mesh's row
// is one chain of row -> ids -> neighbours' rows -> atomic -> append.  The team's barrier at its end.
template <typename Tm>
__device__ __forceinline__ bool search_level(const FeatWork &w, SearchRow *const front[2], SearchRow *huge, int nf,
                                             int L, const Tm &tm, AncShared &sm) {
    const int lane = threadIdx.x & 31;
    const SearchRow *const fin = front[L & 1];
    SearchRow *const fout = front[(L + 1) & 1];
    int *const nout = tm.first(&sm.cnt[(L + 1) % 3]);
    int *const nhuge = tm.first(&sm.nhuge[L & 1]);
    const int d = L + 1;
    if (tm.is_first() && threadIdx.x == 0) {  // last read before the previous level's barrier
        sm.cnt[(L + 2) % 3] = 0;
        sm.nhuge[(L + 1) & 1] = 0;
    }
    for (int i0 = tm.warp() * 16; i0 < nf; i0 += tm.threads() / 2) {
        const int i = i0 + (lane >> 1);
        SearchRow r;
        r.start = 0;
        r.len = 0;
        if (i < nf) r = load_row(fin + i);
        const bool big = r.len > kAncRow;
        const int n = big ? 0 : r.len, most = __reduce_max_sync(DMOLP_FULL_MASK, n);
        for (int c = (lane & 1) * 8; c - (lane & 1) * 8 < most; c += 16) {
            int u[8];
            SearchRow x[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) u[q] = c + q < n ? __ldg(w.col + r.start + c + q) : -1;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                x[q].dist = 0;
                if (u[q] >= 0) x[q] = load_row(w.row + u[q]);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (x[q].dist > d) x[q].dist = atomicMin(&w.row[u[q]].dist, d);
            int cnt = 0;
#pragma unroll
            for (int q = 0; q < 8; ++q) cnt += x[q].dist > d;
            int incl = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
                if (lane >= o) incl += y;
            }
            int base = 0;
            if (lane == 31 && incl) base = atomicAdd(nout, incl);
            int at = __shfl_sync(DMOLP_FULL_MASK, base, 31) + incl - cnt;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (x[q].dist > d) fout[at++] = x[q];
        }
        for (unsigned m = __ballot_sync(DMOLP_FULL_MASK, big && !(lane & 1)); m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            const int64_t s = __shfl_sync(DMOLP_FULL_MASK, r.start, l);
            const int len = __shfl_sync(DMOLP_FULL_MASK, r.len, l);
            if (len > kHugeRow) {
                if (lane == l) huge[atomicAdd(nhuge, 1)] = r;
            } else {
                search_arcs(w, s, s + len, d, nout, fout);
            }
        }
    }
    if (!tm.sync()) return false;
    const int nh = *nhuge;
    if (nh > 0) {  // uniform over the team
        for (int i = 0; i < nh; ++i) {
            const SearchRow r = load_row(huge + i);
            const int64_t s = r.start, e = s + r.len;
            for (int64_t c = s + (int64_t)tm.warp() * 512; c < e; c += (int64_t)tm.threads() * 16)
                search_arcs(w, c, c + 512 < e ? c + 512 : e, d, nout, fout);
        }
        if (!tm.sync()) return false;
    }
    return true;
}

template <typename Tm>
__device__ void run_anchors(const FeatWork &w, int ii, const Tm &tm, AncSmem &sm, AncShared &sh) {
    const Inst I = w.inst[ii];
    const int vb = (int)I.vbase, nv = I.nv;
    SearchRow *const front[2] = {w.front0 + vb, w.front1 + vb};
    SearchRow *const huge = w.huge + vb;
    const bool lead = tm.is_first() && threadIdx.x == 0;
    if (nv == 0) {  // uniform over the team
        if (lead)
            for (int j = 0; j < kAnchors; ++j) w.anchor[j * w.ninst + ii] = -1;
        return;
    }
    for (int i = tm.thread(); i < nv; i += tm.threads()) {
        SearchRow r;
        r.start = w.off[vb + i];
        r.len = (int)(w.off[vb + i + 1] - r.start);
        r.dist = INT_MAX;  // not reached
        w.row[vb + i] = r;
    }
    if (!tm.sync()) return;
    for (int j = 0; j < kAnchors; ++j) {
        // the next anchor: maximum degree, then maximum distance to the anchors so far; lowest id on ties
        unsigned long long key = 0;
        for (int i = tm.thread(); i < nv; i += tm.threads()) {
            const int x = j == 0 ? w.row[vb + i].len : w.row[vb + i].dist;
            if (j > 0 && x == INT_MAX) continue;
            const unsigned long long c = ((unsigned long long)(unsigned)x << 32) | (0xFFFFFFFFu - (unsigned)i);
            key = c > key ? c : key;
        }
        if (!anchor_max(key, j, tm, sm, sh)) return;
        const int a = vb + (int)(0xFFFFFFFFu - (unsigned)(key & 0xFFFFFFFFull));
        if (lead) {
            w.anchor[j * w.ninst + ii] = a;
            SearchRow r = w.row[a];
            r.dist = 0;
            w.row[a] = r;
            front[0][0] = r;
            sh.cnt[1] = sh.cnt[2] = 0;
            sh.nhuge[0] = sh.nhuge[1] = 0;
        }
        if (!tm.sync()) return;
        int nf = 1, L = 0;
        while (nf > 0) {
            if (!search_level(w, front, huge, nf, L, tm, sh)) return;
            nf = *tm.first(&sh.cnt[(L + 1) % 3]);
            ++L;
        }
        if (j == 0 && lead) w.ecc[ii] = L - 1;  // the first anchor's eccentricity
        if (!tm.sync()) return;  // no count is cleared for the next search while it is read
    }
}

__global__ void __launch_bounds__(kAncThreads) k_anchors(FeatWork w, const int32_t *order, int n, int *next) {
    __shared__ AncSmem sm;
    const CtaTeam<kAncThreads> tm;
    for (;;) {
        if (threadIdx.x == 0) sm.inst = atomicAdd(next, 1);
        __syncthreads();
        const int q = sm.inst;
        __syncthreads();
        if (q >= n) break;
        run_anchors(w, order[q], tm, sm, sm.sh);
    }
}

__global__ void __launch_bounds__(kAncThreads) k_anchors_team(FeatWork w, const int32_t *order) {
    __shared__ AncSmem sm;
    const ClusterTeam<kAncThreads> tm;
    run_anchors(w, order[blockIdx.x / tm.size()], tm, sm, sm.sh);
    tm.sync();  // no CTA leaves while its counters are read
}

// Teams of CTAs [start[i], start[i + 1]) of one cooperative launch, team i on graph order[i].
struct GridTeams {
    int n, start[kGridTeams + 1];
    AncShared *sh;
    int *err;
    unsigned int polls;
};

__global__ void __launch_bounds__(kAncThreads) k_anchors_grid(FeatWork w, const int32_t *order, GridTeams t) {
    __shared__ AncSmem sm;
    int i = 0;
    while (i + 1 < t.n && (int)blockIdx.x >= t.start[i + 1]) ++i;
    const GridTeam<kAncThreads> tm = {&t.sh[i].word, t.err, t.polls, t.start[i + 1] - t.start[i],
                                      (int)blockIdx.x - t.start[i]};
    run_anchors(w, order[i], tm, sm, t.sh[i]);
}

// ------------------------------------------------------------------------------------ per-vertex passes
__device__ __forceinline__ int inst_of(const Inst *inst, int ninst, int v) {  // the last with vbase <= v
    int lo = 0, hi = ninst;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (inst[mid].vbase <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The graph of every vertex.
__global__ void k_vinst(const FeatWork w) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < w.nv; v += gridDim.x * blockDim.x)
        w.vinst[v] = inst_of(w.inst, w.ninst, v);
}

// 1 / deg as a float.  (float)(1.0 / (double)deg) equals the float division while deg is exact in a float: a
// quotient of 24-bit numbers rounded to 53 bits first rounds to the same float (53 >= 2 * 24 + 2).
__device__ __forceinline__ float inv_degree(int64_t deg) {
    if (deg <= 0) return 0.f;
    return deg <= (int64_t(1) << 24) ? __fdiv_rn(1.f, (float)deg) : (float)(1.0 / (double)deg);
}

// Random walk state: P (landing probabilities, 8 channels), Q = P / deg.  Eight lanes per vertex.
__global__ void k_rw_init(const FeatWork w) {
    const int64_t n = (int64_t)w.nv * 8;
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
        const int v = (int)(x >> 3), c = (int)(x & 7);
        const float p = w.anchor[c * w.ninst + w.vinst[v]] == v ? 1.f : 0.f;
        w.P0[x] = p;
        w.Q0[x] = __fmul_rn(p, inv_degree(w.off[v + 1] - w.off[v]));
    }
}

// One lazy step of a channel: the sum s over the neighbours' Q, the old P.
__device__ __forceinline__ void rw_next(float s, float p, float inv, float &P, float &Q) {
    P = __fadd_rn(__fmul_rn(0.5f, p), __fmul_rn(0.5f, s));
    Q = __fmul_rn(P, inv);
}

// One lazy step.  Blocks of a long row, the neighbours' Q staged 256 at a time in shared memory by
// all threads while one lane per channel adds the previous tile in row order (the sum is a chain of additions:
// four cycles an arc is its floor).  Other blocks: a chunk each, eight lanes (channels) per vertex, sixteen
// arcs in flight.
__global__ void __launch_bounds__(256) k_rw_step(const FeatWork w, const float *__restrict__ Pin,
                                                 const float *__restrict__ Qin, float *__restrict__ Pout,
                                                 float *__restrict__ Qout) {
    __shared__ float4 tile[2][256][2];
    const Chunk ch = w.chunks[blockIdx.x];
    if (ch.n == 0) {
        const int v = ch.v0;
        const int64_t b = w.off[v], e = w.off[v + 1];
        float4 x0 = make_float4(0, 0, 0, 0), x1 = x0;
        auto load = [&](int64_t j) {
            x0 = x1 = make_float4(0, 0, 0, 0);
            if (j < e) {
                const float4 *q = reinterpret_cast<const float4 *>(Qin + (size_t)__ldg(w.col + j) * 8);
                x0 = q[0];
                x1 = q[1];
            }
        };
        load(b + threadIdx.x);
        float s = 0.f;
        int par = 0;
        for (int64_t j0 = b; j0 < e; j0 += 256, par ^= 1) {
            tile[par][threadIdx.x][0] = x0;
            tile[par][threadIdx.x][1] = x1;
            __syncthreads();  // the tile is full; the other one is no longer read (its sum ended before this)
            load(j0 + 256 + threadIdx.x);
            if (threadIdx.x < 8) {
                const float *t = reinterpret_cast<const float *>(tile[par]) + threadIdx.x;
                const int n = e - j0 < 256 ? (int)(e - j0) : 256;
                int i = 0;
                for (; i + 16 <= n; i += 16) {
                    float y[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) y[q] = t[(i + q) * 8];
#pragma unroll
                    for (int q = 0; q < 16; ++q) s = __fadd_rn(s, y[q]);
                }
                for (; i < n; ++i) s = __fadd_rn(s, t[i * 8]);
            }
        }
        if (threadIdx.x < 8) {
            const size_t x = (size_t)v * 8 + threadIdx.x;
            rw_next(s, Pin[x], inv_degree(e - b), Pout[x], Qout[x]);
        }
        return;
    }
    const int c = threadIdx.x & 7, lane = threadIdx.x & 31;
    for (int i0 = (int)(threadIdx.x >> 5) * 4; i0 < ch.n; i0 += 32) {  // four vertices per warp
        const int i = i0 + (lane >> 3);
        const int v = ch.v0 + (i < ch.n ? i : 0);
        const int64_t b = w.off[v];
        const int64_t deg = w.off[v + 1] - b;
        const bool mine = i < ch.n && deg <= kLongRow;
        const int len = mine ? (int)deg : 0, most = __reduce_max_sync(DMOLP_FULL_MASK, len);
        const float p = mine ? Pin[(size_t)v * 8 + c] : 0.f;
        float s = 0.f;
        for (int j = 0; j < most; j += kWalkU) {  // arcs past the row's end add +0 to a sum that is never negative
            int u[kWalkU / 8];
            float y[kWalkU];
#pragma unroll
            for (int q = 0; q < kWalkU / 8; ++q) u[q] = j + 8 * q + c < len ? __ldg(w.col + b + j + 8 * q + c) : -1;
#pragma unroll
            for (int q = 0; q < kWalkU; ++q) {
                const int x = __shfl_sync(DMOLP_FULL_MASK, u[q >> 3], q & 7, 8);
                y[q] = x >= 0 ? Qin[(size_t)x * 8 + c] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < kWalkU; ++q) s = __fadd_rn(s, y[q]);
        }
        if (mine) {
            const size_t x = (size_t)v * 8 + c;
            rw_next(s, p, inv_degree(len), Pout[x], Qout[x]);
        }
    }
}

// log landing probabilities, their per-graph sums and sums of squares (double): a block per chunk, eight lanes
// per vertex, one atomic per block and sum.  A graph that walked T steps left its probabilities in P0 (T even)
// or P1 (T odd): steps alternate the two buffers.
__global__ void __launch_bounds__(256) k_rw_log(const FeatWork w) {
    __shared__ double part[8][16];
    const Chunk ch = w.chunks[blockIdx.x];
    if (ch.n == 0) return;  // a long row: its vertex is in a chunk, too
    const int c = threadIdx.x & 7, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *P = (min(max(w.ecc[ch.inst], 1), kTMax) & 1) ? w.P1 : w.P0;
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x >> 3; i < ch.n; i += 32) {
        const size_t v = (size_t)(ch.v0 + i);
        const float L = logf(fmaxf(P[v * 8 + c], kPFloor));
        w.Xf[v * 16 + 2 + c] = L;
        a += (double)L;
        b += (double)L * (double)L;
    }
    for (int o = 8; o < 32; o <<= 1) {
        a += __shfl_xor_sync(DMOLP_FULL_MASK, a, o);
        b += __shfl_xor_sync(DMOLP_FULL_MASK, b, o);
    }
    if (lane < 8) {
        part[warp][c] = a;
        part[warp][8 + c] = b;
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        double t = 0.0;
        for (int i = 0; i < 8; ++i) t += part[i][threadIdx.x];
        atomicAdd(&w.stats[(size_t)ch.inst * 16 + threadIdx.x], t);
    }
}

// The features of a chunk's vertices, float and (layer 1's input) bf16: four lanes per vertex, four columns each.
__global__ void __launch_bounds__(256) k_feat_final(const FeatWork w) {
    __shared__ float mu[8], sd[8];
    const Chunk ch = w.chunks[blockIdx.x];
    if (ch.n == 0) return;
    const Inst I = w.inst[ch.inst];
    if (threadIdx.x < 8) {
        const double n = (double)I.nv, m = w.stats[(size_t)ch.inst * 16 + threadIdx.x] / n;
        const float s = (float)sqrt(fmax(w.stats[(size_t)ch.inst * 16 + 8 + threadIdx.x] / n - m * m, 0.0));
        mu[threadIdx.x] = (float)m;
        sd[threadIdx.x] = s > 0.f ? s : 1.f;
    }
    __syncthreads();
    const float mdeg = I.narcs > 0 ? (float)((double)I.narcs / (double)I.nv) : 1.f;
    const int q = threadIdx.x & 3;
    for (int i = threadIdx.x >> 2; i < ch.n; i += 64) {
        const size_t v = (size_t)(ch.v0 + i);
        float4 *xp = reinterpret_cast<float4 *>(w.Xf + v * 16) + q;
        const float4 raw = q < 3 ? *xp : make_float4(0, 0, 0, 0);
        const float in[4] = {raw.x, raw.y, raw.z, raw.w};
        float x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int col = 4 * q + t, j = col - 2;
            x[t] = j >= 0 && j < 8 ? __fdiv_rn(__fsub_rn(in[t], mu[j & 7]), sd[j & 7]) : 0.f;
            if (col == 10) x[t] = __fdiv_rn((float)I.k, 64.f);
        }
        if (q == 0) {
            const int64_t deg = w.off[v + 1] - w.off[v];
            x[0] = __fdiv_rn((float)deg, mdeg);
            x[1] = log1pf((float)deg);
        }
        *xp = make_float4(x[0], x[1], x[2], x[3]);
        const __nv_bfloat162 h0 = __floats2bfloat162_rn(x[0], x[1]), h1 = __floats2bfloat162_rn(x[2], x[3]);
        __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(w.X + v * w.ldx + 4 * q);
        o[0] = h0;
        o[1] = h1;
    }
}

__global__ void k_to_input(const float *Xf, int nv, __nv_bfloat16 *X, int ldx) {
    const int64_t n = (int64_t)nv * 4;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 x = reinterpret_cast<const float4 *>(Xf)[i];
        __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(X + (size_t)(i >> 2) * ldx + 4 * (int)(i & 3));
        o[0] = __floats2bfloat162_rn(x.x, x.y);
        o[1] = __floats2bfloat162_rn(x.z, x.w);
    }
}

int grid_for(int64_t n, int num_sms) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)num_sms * 16));
}

int anchors_max_team() {
    for (int c = batch::kMaxTeam; c > 1; c >>= 1) {
        int n = 0;
        if (batch::max_clusters(k_anchors_team, c, kAncThreads, &n) && n > 0) return c;
    }
    return 1;
}

}  // namespace

int features(const FeatWork &w, const batch::View &b, cudaStream_t s) {
    if (w.nv <= 0) return 0;
    const int g = grid_for(w.nv, b.num_sms);
    cudaMemsetAsync(w.next, 0, sizeof(int), s);
    cudaMemsetAsync(w.ecc, 0, sizeof(int32_t) * w.ninst, s);
    cudaMemsetAsync(w.stats, 0, sizeof(double) * 16 * w.ninst, s);
    k_vinst<<<g, 256, 0, s>>>(w);
    {
        std::vector<int32_t> order = *b.h_order;
        int slots = b.num_sms;
        const int32_t *o = b.order;
        // graphs worth more than a cluster, largest first
        double total = 0;
        for (int32_t i : order) total += (double)((*b.h_inst)[i].narcs + (*b.h_inst)[i].nv);
        GridTeams gt = {};
        for (int32_t i : order) {
            const Inst &I = (*b.h_inst)[i];
            const int c = (int)((double)(I.narcs + I.nv) * b.num_sms / total);
            if (gt.n == kGridTeams || c <= kGridShare || I.nv <= c * kAncThreads) break;
            gt.start[gt.n + 1] = gt.start[gt.n] + std::min(c, slots);
            slots -= std::min(c, slots);
            ++gt.n;
        }
        if (gt.n > 0) {
            static_assert(sizeof(AncShared) * kGridTeams <= kFeatSharedBytes, "the teams' counters fit their buffer");
            gt.sh = reinterpret_cast<AncShared *>(w.shared);
            gt.err = w.err;
            gt.polls = w.polls;
            cudaMemsetAsync(w.shared, 0, kFeatSharedBytes, s);
            cudaEventRecord(b.fork->begin, s);  // the other graphs run next to them
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)gt.start[gt.n]);
            cfg.blockDim = dim3(kAncThreads);
            cfg.stream = s;
            cudaLaunchAttribute at;
            at.id = cudaLaunchAttributeCooperative;
            at.val.cooperative = 1;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            const cudaError_t le = cudaLaunchKernelEx(&cfg, k_anchors_grid, w, o, gt);
            if (le != cudaSuccess) return (int)le;
            order.erase(order.begin(), order.begin() + gt.n);
            o += gt.n;
            slots = std::max(slots, 1);
        }
        // (next to such teams every class runs on its own side stream, which the clusters of 16 have not)
        const int most = anchors_max_team();
        const batch::TeamPlan plan =
            batch::team_sizes(*b.h_inst, order, slots, kAncThreads, gt.n > 0 ? std::min(most, batch::kMaxTeam / 2) : most);
        const int j1 = batch::kTeamClasses - 1, n1 = plan.n[j1];
        if (gt.n > 0) {
            for (int j = 1; j <= j1; ++j)
                if (plan.n[j] > 0) cudaStreamWaitEvent(b.fork->side[j - 1], b.fork->begin, 0);
        } else {
            b.fork->open(plan, s);
        }
        auto on = [&](int j) { return gt.n > 0 ? b.fork->side[j - 1] : b.fork->stream(plan, j, s); };
        for (int j = 0, c = batch::kMaxTeam; c > 1; ++j, c >>= 1) {
            if (plan.n[j] > 0) batch::launch_cluster(k_anchors_team, plan.n[j], c, kAncThreads, on(j), w, o);
            o += plan.n[j];
        }
        if (n1 > 0) k_anchors<<<std::min(b.num_sms, n1), kAncThreads, 0, on(j1)>>>(w, o, n1, w.next);
        if (gt.n > 0) {
            for (int j = 1; j <= j1; ++j)
                if (plan.n[j] > 0) {
                    cudaEventRecord(b.fork->end[j - 1], b.fork->side[j - 1]);
                    cudaStreamWaitEvent(s, b.fork->end[j - 1], 0);
                }
        } else {
            b.fork->close(plan, s);
        }
    }
    std::vector<int32_t> ecc(w.ninst);
    cudaMemcpyAsync(ecc.data(), w.ecc, sizeof(int32_t) * w.ninst, cudaMemcpyDeviceToHost, s);
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return (int)e;
    for (int32_t &x : ecc) x = std::min(std::max(x, 1), kTMax);
    // The walk's order: graphs by descending steps; step t launches the first walking[t] units.
    std::vector<int32_t> by;
    for (int i = 0; i < w.ninst; ++i)
        if ((*b.h_inst)[i].nv > 0) by.push_back(i);
    std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return ecc[x] > ecc[y]; });
    std::vector<Chunk> chunks;
    std::vector<int> walking(by.empty() ? 0 : ecc[by[0]], 0);
    for (int32_t i : by) {
        const Inst &I = (*b.h_inst)[i];
        auto lr = std::lower_bound(b.h_longrow->begin(), b.h_longrow->end(), (int32_t)I.vbase);
        for (; lr != b.h_longrow->end() && *lr < I.vbase + I.nv; ++lr) chunks.push_back(Chunk{*lr, 0, i});
        for (int v = 0; v < I.nv; v += kChunkV)
            chunks.push_back(Chunk{(int)I.vbase + v, std::min(kChunkV, I.nv - v), i});
        for (int t = 0; t < ecc[i]; ++t) walking[t] = (int)chunks.size();
    }
    cudaMemcpyAsync(w.chunks, chunks.data(), chunks.size() * sizeof(Chunk), cudaMemcpyHostToDevice, s);
    k_rw_init<<<grid_for((int64_t)w.nv * 8, b.num_sms), 256, 0, s>>>(w);
    float *P = w.P0, *Q = w.Q0, *P2 = w.P1, *Q2 = w.Q1;
    for (int n : walking) {
        k_rw_step<<<n, 256, 0, s>>>(w, P, Q, P2, Q2);
        std::swap(P, P2);
        std::swap(Q, Q2);
    }
    k_rw_log<<<(int)chunks.size(), 256, 0, s>>>(w);
    k_feat_final<<<(int)chunks.size(), 256, 0, s>>>(w);
    return (int)cudaGetLastError();
}

void features_to_input(const float *Xf, int nv, __nv_bfloat16 *X, int ldx, int num_sms, cudaStream_t s) {
    k_to_input<<<grid_for((int64_t)nv * 4, num_sms), 256, 0, s>>>(Xf, nv, X, ldx);
}

}  // namespace mpnn
}  // namespace dmolp
