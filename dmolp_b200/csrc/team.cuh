// Teams of CTAs that work on one graph of a batch: a single CTA, or a thread-block cluster whose CTAs share
// counters through distributed shared memory.  The kernels are written once against this interface.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace dmolp {
namespace batch {

// One CTA.
template <int NT>
struct CtaTeam {
    __device__ __forceinline__ constexpr int size() const { return 1; }
    __device__ __forceinline__ constexpr bool is_first() const { return true; }
    __device__ __forceinline__ constexpr int rank_of() const { return 0; }
    __device__ __forceinline__ int thread() const { return threadIdx.x; }
    __device__ __forceinline__ constexpr int threads() const { return NT; }
    __device__ __forceinline__ int warp() const { return threadIdx.x >> 5; }
    __device__ __forceinline__ bool sync() const {
        __syncthreads();
        return true;
    }
    template <typename T>
    __device__ __forceinline__ T *at(T *p, int) const {
        return p;
    }
    template <typename T>
    __device__ __forceinline__ T *first(T *p) const {
        return p;
    }
};

// A cluster.  at(p, r): the address in CTA r's shared memory of what p is in this CTA's.  Warps are numbered
// round-robin over the CTAs, so short lists spread over all SMs.  sync() is the cluster barrier: it orders the
// team's global and shared accesses on both sides (release / acquire at cluster scope).
template <int NT>
struct ClusterTeam {
    int n, rank;
    __device__ __forceinline__ ClusterTeam()
        : n((int)cooperative_groups::this_cluster().num_blocks()),
          rank((int)cooperative_groups::this_cluster().block_rank()) {}
    __device__ __forceinline__ int size() const { return n; }
    __device__ __forceinline__ bool is_first() const { return rank == 0; }
    __device__ __forceinline__ int rank_of() const { return rank; }
    __device__ __forceinline__ int warp() const { return (int)(threadIdx.x >> 5) * n + rank; }
    __device__ __forceinline__ int threads() const { return NT * n; }
    __device__ __forceinline__ int thread() const { return warp() * 32 + (int)(threadIdx.x & 31); }
    __device__ __forceinline__ bool sync() const {
        cooperative_groups::this_cluster().sync();
        return true;
    }
    template <typename T>
    __device__ __forceinline__ T *at(T *p, int r) const {
        return cooperative_groups::this_cluster().map_shared_rank(p, r);
    }
    template <typename T>
    __device__ __forceinline__ T *first(T *p) const {
        return at(p, 0);
    }
};

// Some of the CTAs of a cooperative launch (all resident), for graphs that are worth more CTAs than a cluster has.
// They share no shared memory: the team's counters are one object in global memory, which first(p) leaves as it is,
// and code for this team keeps nothing else per CTA in it.  sync() is a barrier on one word (arrive_and_wait).  It
// returns false when the wait gave up after `polls` polls, or another CTA's did (*err is then set): the caller leaves
// the kernel at once.
template <int NT>
struct GridTeam {
    unsigned int *word;
    int *err;
    unsigned int polls;
    int n, rank;
    __device__ __forceinline__ int size() const { return n; }
    __device__ __forceinline__ bool is_first() const { return rank == 0; }
    __device__ __forceinline__ int rank_of() const { return rank; }
    __device__ __forceinline__ int warp() const { return (int)(threadIdx.x >> 5) * n + rank; }
    __device__ __forceinline__ int threads() const { return NT * n; }
    __device__ __forceinline__ int thread() const { return warp() * 32 + (int)(threadIdx.x & 31); }
    __device__ __forceinline__ bool sync() const {
        bool pass = true;
        __syncthreads();
        if (threadIdx.x == 0) {
            pass = arrive_and_wait(word, (unsigned int)n, rank == 0, polls, err);
            if (!pass) atomicExch(err, 1);
        }
        return __syncthreads_and(pass);
    }
    template <typename T>
    __device__ __forceinline__ T *first(T *p) const {
        return p;
    }
};

// Slots for the lanes with pred, taken from a counter with one atomic per warp (all lanes call it).
__device__ __forceinline__ int warp_push(int *ctr, bool pred) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(DMOLP_FULL_MASK, pred);
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(ctr, __popc(m));
    base = __shfl_sync(DMOLP_FULL_MASK, base, 0);
    return base + __popc(m & ((1u << lane) - 1));
}

// Maximum of a 64-bit key over the team (every thread passes its own; the result in every thread).  Two
// barriers of the team; wbest[NT / 32] and cbest are the CTA's scratch.
template <int NT, typename Tm>
__device__ __forceinline__ unsigned long long team_max(unsigned long long x, const Tm &tm, unsigned long long *wbest,
                                                       unsigned long long *cbest) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(DMOLP_FULL_MASK, x, o);
        x = y > x ? y : x;
    }
    if ((threadIdx.x & 31) == 0) wbest[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long r = 0;
        for (int i = 0; i < NT / 32; ++i) r = wbest[i] > r ? wbest[i] : r;
        *cbest = r;
    }
    tm.sync();
    unsigned long long r = 0;
    for (int c = 0; c < tm.size(); ++c) {
        const unsigned long long y = *tm.at(cbest, c);
        r = y > r ? y : r;
    }
    tm.sync();  // cbest may be rewritten
    return r;
}

// Visit the n vertices vid(i), i in [0, n).  Every thread of the team calls it.  small(active, v, s, e) is
// called by all lanes of a warp (active marks the lanes that own a short row [s, e)); rows with
// is_big(v, s, e) are passed one by one to wide(v, s, e), called by the whole warp.
template <typename Tm, typename Vid, typename Big, typename Small, typename Wide>
__device__ __forceinline__ void visit(const int64_t *off, const Tm &tm, int n, Vid vid, Big is_big, Small small,
                                      Wide wide) {
    const int lane = threadIdx.x & 31;
    for (int i0 = tm.warp() * 32; i0 < n; i0 += tm.threads()) {
        const int i = i0 + lane;
        int v = -1;
        int64_t s = 0, e = 0;
        if (i < n) {
            v = vid(i);
            s = off[v];
            e = off[v + 1];
        }
        const bool big = v >= 0 && is_big(v, s, e);
        small(v >= 0 && !big, v, s, e);
        unsigned m = __ballot_sync(DMOLP_FULL_MASK, big);
        while (m) {
            const int l = __ffs(m) - 1;
            m &= m - 1;
            wide(__shfl_sync(DMOLP_FULL_MASK, v, l), __shfl_sync(DMOLP_FULL_MASK, s, l),
                 __shfl_sync(DMOLP_FULL_MASK, e, l));
        }
    }
}

// The per-part radix select of a team: records of 6-bit digits, most significant first.
constexpr int kDigitBits = 6;
constexpr int kDigits = 1 << kDigitBits;
constexpr int kMaxPass = 12;   // 6-bit digits of a key of at most 62 bits, and one more
constexpr int kOwnShift = 58;  // a record's part sits above its key (when the key has at most 58 bits)

// One digit's cut: per part p < k (one warp of the team each, 2 bins per lane) the digit where the running
// count over the team's histograms crosses need[p].  To every CTA: below[p] = digits under it are selected,
// keep[p] = the digit whose records stay open for the next pass (-1: none).  need[p] becomes what is left to
// take from those; it is read and written by the part's warp alone.
template <typename Tm>
__device__ __forceinline__ void cut_digit(const Tm &tm, int k, int *hist, int *need, int *below, int *keep) {
    const int lane = threadIdx.x & 31;
    for (int p = tm.warp(); p < k; p += tm.threads() / 32) {
        int c0 = 0, c1 = 0;
        for (int r = 0; r < tm.size(); ++r) {
            const int2 h = *reinterpret_cast<const int2 *>(tm.at(hist + p * kDigits + 2 * lane, r));
            c0 += h.x;
            c1 += h.y;
        }
        const int sum = c0 + c1;
        int incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
            if (lane >= o) incl += y;
        }
        const int total = __shfl_sync(DMOLP_FULL_MASK, incl, 31);
        const int nd = need[p];
        int b = -1, kp = -1, left = 0;
        if (nd <= 0) {
            b = 0;
        } else if (nd >= total) {
            b = kDigits;
        } else {
            const int ex0 = incl - sum, in0 = ex0 + c0, in1 = in0 + c1;
            int d = -1, r = 0, cnt = 0;
            if (ex0 < nd && nd <= in0) {
                d = 2 * lane;
                r = nd - ex0;
                cnt = c0;
            } else if (in0 < nd && nd <= in1) {
                d = 2 * lane + 1;
                r = nd - in0;
                cnt = c1;
            }
            if (d >= 0) {
                b = r == cnt ? d + 1 : d;
                kp = r == cnt ? -1 : d;
                left = r == cnt ? 0 : r;
            }
        }
        const int src = __ffs(__ballot_sync(DMOLP_FULL_MASK, b >= 0)) - 1;
        b = __shfl_sync(DMOLP_FULL_MASK, b, src);
        kp = __shfl_sync(DMOLP_FULL_MASK, kp, src);
        left = __shfl_sync(DMOLP_FULL_MASK, left, src);
        if (lane == 0) need[p] = left;
        for (int r = lane; r < tm.size(); r += 32) {
            *tm.at(below + p, r) = b;
            *tm.at(keep + p, r) = kp;
        }
    }
}

// Whether any part still has open records (the same in every thread of the team).
__device__ __forceinline__ bool any_open(int k, const int *keep) {
    const int lane = threadIdx.x & 31;
    return __any_sync(DMOLP_FULL_MASK, (lane < k && keep[lane] >= 0) || (lane + 32 < k && keep[lane + 32] >= 0));
}

}  // namespace batch
}  // namespace dmolp
