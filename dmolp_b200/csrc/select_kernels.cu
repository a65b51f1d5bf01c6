// The LP's window selections: the radix select (select_radix.cuh) as a kernel of its own, and the degree-bin
// selection.
#include "select_radix.cuh"

namespace dmolp {
namespace {

__global__ void __launch_bounds__(kSelThreads, 1) k_select(SelArgs a) {
    if (a.stopped && *a.stopped) return;  // the same for every block: all return, no barrier is left open
    select_body<true>(a, *a.n_dev, nullptr);
}

// ------------------------------------------------------------------------------------------------------
// Degree-bin window selection (LP, at most kDegSelMaxK labels).
//
// Per label p the window takes need_p = min(n_p, ceil(e^(-t/5) n_p)) of the label's n_p boundary records:
// the smallest degrees first, or the largest first when RE[p] > 1, ids ascending among equal degrees
// (gpu_lp_boundary.cu:244, 282-300).  The boundary test has counted every label's records per degree
// superbin (dsel_bin, Buffers::dsup).  One cooperative launch, one block per SM, ONE grid barrier:
//   0. every block finds, per label, the superbin where the running count in the label's order reaches
//      need_p; records of the superbins before it are taken, the rest of that superbin is partial;
//   1. each warp walks its own contiguous range of record slots in order: taken records go to the window;
//      records of a partial superbin of degree < 2048 go to the warp's list (label and key, in slot order)
//      and into the block's fine-bin counts (stored per block in dcntb, summed into dfine); the keys of those
//      of degree >= 2048 to their label's segment of a tail list (segments sized by the superbin counts) and
//      into dfine;
//   -- grid barrier --
//   2. every block finds, per label, the fine bin of the partial superbin where the count reaches the rest
//      of the need.  Below degree 2048 a fine bin is a single degree, and record slots hold the vertices of
//      one degree in ascending id order (slots follow the degree classes, ids ascending inside a class), so
//      a record of the partial fine bin is taken when fewer than the rest of the need precede it: in the
//      blocks before this one (dcntb), in the warps before this one, in its warp's list before it.  Above,
//      block p sorts label p's tail keys of the partial fine bin (degree, then id) and takes the first ones.
// ------------------------------------------------------------------------------------------------------
constexpr int kDsThreads = 1024;
constexpr int kDsWarps = kDsThreads / 32;
constexpr int kDsU = 2;          // record slots per lane and step of the first walk
constexpr int kDsTieCap = 4096;  // a label's coarse tied records ranked in shared memory (more: from global)

struct DegSelArgs {
    const int32_t *seg;        // bown: label of a boundary record, -1 for an empty slot
    const uint64_t *key;       // bkey: (dk << ibits) | v
    const int *n_dev;          // record slots
    int32_t *lists;            // the warps' lists of partial-superbin records below degree 2048: labels ...
    uint64_t *lkeys;           // ... and keys (the same positions)
    uint64_t *tail;            // keys of partial-superbin records of degree >= 2048, one segment per label
    int *tcnt, *tcnt_next;     // [nseg] tail records per label (this iteration / the next one's, cleared here)
    unsigned int *dsup;        // [nseg * kDsBins] from the boundary test; cleared here after the barrier
    unsigned int *dfine;       // [nseg * kDsFine] fine counts of this iteration's partial superbins
    unsigned int *dfine_next;  // the other parity's buffer, cleared here for the next iteration
    unsigned int *dcntb;       // [gridDim.x * nseg * kDsFine]
    int nseg;
    unsigned int polls;
    LpControl *ctl;
    const int *stopped;
    SplitArgs sp;
};

// Dynamic shared memory of k_select_deg for nseg labels.
__host__ __device__ constexpr size_t ds_smem_bytes(int nseg) {
    return (size_t)kDsTieCap * 8 + (size_t)10 * nseg * 4 + (size_t)nseg * kDsFine * 4 +
           (size_t)2 * kDsWarps * nseg * 4 + (size_t)kDsWarps * 4 * kStage * 4;
}

// Order position of superbin / fine bin x in a label's order (descending degree when dir).
__device__ __forceinline__ int ds_ord(int x, int n, int dir) { return dir ? n - 1 - x : x; }

// Running-count crossing over `per` consecutive order positions per lane (all lanes): the position where
// the count reaches need (0 < need < total), the records before it and its count.
template <int PER, typename C>
__device__ __forceinline__ void ds_cross(int need, C cnt_at, int lane, int &pos, int &before, int &count) {
    unsigned int c[PER], sum = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        c[j] = cnt_at(lane * PER + j);
        sum += c[j];
    }
    unsigned int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
        if (lane >= o) incl += y;
    }
    unsigned int run = incl - sum;
    int fpos = -1, fbefore = 0, fcount = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (run < (unsigned)need && (unsigned)need <= run + c[j]) {
            fpos = lane * PER + j;
            fbefore = (int)run;
            fcount = (int)c[j];
        }
        run += c[j];
    }
    const unsigned m = __ballot_sync(DMOLP_FULL_MASK, fpos >= 0);
    const int src = m ? __ffs(m) - 1 : 0;
    pos = __shfl_sync(DMOLP_FULL_MASK, fpos, src);
    before = __shfl_sync(DMOLP_FULL_MASK, fbefore, src);
    count = __shfl_sync(DMOLP_FULL_MASK, fcount, src);
}

__global__ void __launch_bounds__(kDsThreads, 1) k_select_deg(DegSelArgs a) {
    if (a.stopped && *a.stopped) return;  // the same for every block: all return, no barrier is left open
    extern __shared__ __align__(16) unsigned char ds_smem[];
    const int nseg = a.nseg, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1;
    uint64_t *s_tkey = reinterpret_cast<uint64_t *>(ds_smem);       // [kDsTieCap] keys of this block's coarse ties
    int *s_otake = reinterpret_cast<int *>(s_tkey + kDsTieCap);     // [nseg] superbin order positions below this are taken
    int *s_opart = s_otake + nseg;       // [nseg] order position of the partial superbin, -1 none
    int *s_rem = s_opart + nseg;         // [nseg] records still needed from the partial superbin
    int *s_dir = s_rem + nseg;           // [nseg] 1: largest degree first (RE > 1)
    int *s_kind = s_dir + nseg;          // [nseg] partial superbin: 0 none, 1 one degree, 2 < 2048, 3 coarse
    int *s_toff = s_kind + nseg;         // [nseg] the label's segment of the tail list
    int *s_ftake = s_toff + nseg;        // [nseg] fine order positions below this are taken
    int *s_fpart = s_ftake + nseg;       // [nseg] fine order position of the partial fine bin, -1 none
    int *s_frem = s_fpart + nseg;        // [nseg] records still needed from the partial fine bin
    int *s_pre = s_frem + nseg;          // [nseg] the partial fine bin's records in the blocks before this one
    unsigned int *s_f = reinterpret_cast<unsigned int *>(s_pre + nseg);  // [nseg * kDsFine] this block's
    int *s_wc = reinterpret_cast<int *>(s_f + nseg * kDsFine);  // [kDsWarps * nseg] partial fine bin per warp
    int *s_wrun = s_wc + kDsWarps * nseg;                       // [kDsWarps * nseg] running rank per warp
    int *s_stage = s_wrun + kDsWarps * nseg;                    // [kDsWarps * 4 * kStage] window appends
    __shared__ int s_scnt[kDsWarps][4];
    __shared__ int s_ntie, s_walk1, s_bstar, s_before;
    __shared__ unsigned int s_wsum[kDsWarps];
    __shared__ int s_soff[kDsWarps][4], s_sbase[4];
    __shared__ unsigned long long s_te[kDsWarps], s_ws[kDsWarps];
    int *w_stage = s_stage + wid * 4 * kStage, *w_scnt = s_scnt[wid];
    if (lane < 4) w_scnt[lane] = 0;
    for (int i = threadIdx.x; i < nseg * kDsFine; i += blockDim.x) s_f[i] = 0u;
    for (int i = threadIdx.x; i < kDsWarps * nseg; i += blockDim.x) s_wc[i] = 0;
    if (threadIdx.x == 0) {
        s_ntie = 0;
        s_walk1 = 0;
    }
    // the other parity's fine and tail counts were used by the previous iteration's selection: clear them
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nseg * kDsFine; i += gridDim.x * blockDim.x)
        a.dfine_next[i] = 0u;
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < nseg; i += blockDim.x) a.tcnt_next[i] = 0;
    // ---- 0. per label: the superbin where the need is reached ----
    const double ratio = *a.sp.ratio;
    for (int p = wid; p < nseg; p += kDsWarps) {
        const int n = a.sp.npart[p];
        const int m = (int)ceil(__dmul_rn(ratio, (double)n));  // ceil(e^(-t/5) n), gpu_lp_boundary.cu:296-297
        const int need = m > n ? n : m;
        const int dir = __ldg(a.sp.RE + p) > 1.0 ? 1 : 0;
        int take = need >= n ? kDsBins : 0, part = -1, rem = 0, kind = 0, tsize = 0;
        if (need > 0 && need < n) {
            int pos, before, count;
            ds_cross<(kDsBins + 31) / 32>(need, [&](int o) {
                return o < kDsBins ? __ldcg(a.dsup + p * kDsBins + ds_ord(o, kDsBins, dir)) : 0u;
            }, lane, pos, before, count);
            if (pos < 0) {  // inconsistent counts (never expected): take nothing more
                take = 0;
            } else if (need - before == count) {
                take = pos + 1;
            } else {
                take = pos;
                part = pos;
                rem = need - before;
                const int sb = ds_ord(pos, kDsBins, dir);
                kind = sb < kDsSingle ? 1 : (sb < kDsCoarse0 ? 2 : 3);
                if (kind == 3) tsize = count;
            }
        }
        if (lane == 0) {
            s_otake[p] = take;
            s_opart[p] = part;
            s_rem[p] = rem;
            s_dir[p] = dir;
            s_kind[p] = kind;
            s_toff[p] = tsize;  // the segment sizes, turned into offsets below
        }
    }
    __syncthreads();
    if (wid == 0) {  // exclusive prefix of the tail segment sizes (nseg <= 64: two per lane)
        const int x0 = lane < nseg ? s_toff[lane] : 0, x1 = lane + 32 < nseg ? s_toff[lane + 32] : 0;
        int incl = x0 + x1;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
            if (lane >= o) incl += y;
        }
        const int excl = incl - x0 - x1;
        __syncwarp();
        if (lane < nseg) s_toff[lane] = excl;
        if (lane + 32 < nseg) s_toff[lane + 32] = excl + x0;
    }
    __syncthreads();
    // ---- 1. each warp walks its own contiguous range of record slots ----
    const int n0 = *a.n_dev;
    const int cap = (n0 + gridDim.x - 1) / gridDim.x;
    const int lo = blockIdx.x * cap;
    const int my_n = max(0, min(n0, lo + cap) - lo);
    const int wcap = (my_n + kDsWarps - 1) / kDsWarps;
    const int wlo = lo + min(my_n, wid * wcap), whi = lo + min(my_n, (wid + 1) * wcap);
    int32_t *wlist = a.lists + wlo;  // at most whi - wlo entries: label, and the key in lkeys
    uint64_t *wkey = a.lkeys + wlo;
    int wl = 0;                      // the warp's list length (warp-uniform)
    const int ibits = a.sp.ibits, maxdeg = a.sp.maxdeg;
    const uint64_t vmask = (1ull << ibits) - 1;
    unsigned long long te = 0, ws = 0;
    auto bins_of = [&](uint64_t key, int p, int &o, int &fo) {
        const int dir = s_dir[p];
        const int dk = (int)(key >> ibits);
        const int2 bf = dsel_bin(dir ? maxdeg - dk : dk);
        o = ds_ord(bf.x, kDsBins, dir);
        fo = ds_ord(bf.y, kDsFine, dir);
        return bf;
    };
    // the next step's slots are loaded while this step's are processed
    int np_[kDsU];
    uint64_t nkey[kDsU];
#pragma unroll
    for (int u = 0; u < kDsU; ++u) {
        const int r = wlo + u * 32 + lane;
        np_[u] = r < whi ? a.seg[r] : -1;
        nkey[u] = r < whi ? a.key[r] : 0;
    }
    for (int r0 = wlo; r0 < whi; r0 += 32 * kDsU) {
        int p[kDsU], fb[kDsU];
        uint64_t key[kDsU];
        bool take[kDsU], part[kDsU];
#pragma unroll
        for (int u = 0; u < kDsU; ++u) {
            p[u] = np_[u];
            key[u] = nkey[u];
            const int r = r0 + 32 * kDsU + u * 32 + lane;
            np_[u] = r < whi ? a.seg[r] : -1;
            nkey[u] = r < whi ? a.key[r] : 0;
        }
        bool some = false;
#pragma unroll
        for (int u = 0; u < kDsU; ++u) some |= p[u] >= 0;
        if (!__any_sync(DMOLP_FULL_MASK, some)) continue;  // empty slots only
#pragma unroll
        for (int u = 0; u < kDsU; ++u) {
            take[u] = part[u] = false;
            fb[u] = -1;
            if (p[u] >= 0) {
                int o, fo;
                const int2 bf = bins_of(key[u], p[u], o, fo);
                if (o < s_otake[p[u]]) {
                    take[u] = true;
                } else if (o == s_opart[p[u]]) {
                    part[u] = true;
                    fb[u] = p[u] * kDsFine + bf.y;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kDsU; ++u) {
            // fine counts; a partial superbin of one degree has a single fine bin, so its records are also
            // counted per warp (the ties' ranks need no second walk of the list)
            const bool coarse = part[u] && s_kind[p[u]] == 3;
            if (part[u]) {
                atomicAdd(&s_f[fb[u]], 1u);
                if (s_kind[p[u]] == 1) atomicAdd(&s_wc[wid * nseg + p[u]], 1);
            }
            // records below degree 2048 to the warp's list, in slot order; coarse ones to their label's
            // tail segment (one global atomic per label group of the warp)
            const unsigned mp = __ballot_sync(DMOLP_FULL_MASK, part[u] && !coarse);
            if (part[u] && !coarse) {
                wlist[wl + __popc(mp & below)] = p[u];
                wkey[wl + __popc(mp & below)] = key[u];
            }
            wl += __popc(mp);
            if (__any_sync(DMOLP_FULL_MASK, coarse)) {
                const unsigned mc = __match_any_sync(DMOLP_FULL_MASK, coarse ? p[u] : -1 - lane);
                int q = 0;
                if (coarse && lane == __ffs(mc) - 1) q = atomicAdd(&a.tcnt[p[u]], __popc(mc));
                q = __shfl_sync(DMOLP_FULL_MASK, q, coarse ? __ffs(mc) - 1 : lane);
                if (coarse) a.tail[s_toff[p[u]] + q + __popc(mc & below)] = key[u];
            }
        }
        emit_window<kDsU>(a.sp, take, key, p, vmask, te, ws, w_stage, w_scnt);  // all lanes
    }
    __syncthreads();
    // this block's fine counts: kept per block for the prefixes, summed for the fine decisions
    for (int i = threadIdx.x; i < nseg * kDsFine; i += blockDim.x) {
        const unsigned int v = s_f[i];
        a.dcntb[(size_t)blockIdx.x * nseg * kDsFine + i] = v;
        if (v) atomicAdd(&a.dfine[i], v);
    }
    if (!grid_sync(a.ctl, a.polls, 0)) return;
    // every block has read the superbin counts: clear them for the next boundary test
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nseg * kDsBins; i += gridDim.x * blockDim.x) a.dsup[i] = 0u;
    // ---- 2. per label with a partial superbin: the fine bin where the rest of the need is reached ----
    for (int p = wid; p < nseg; p += kDsWarps) {
        int take = 0, part = -1, rem = 0, pre = 0;
        const int kind = s_kind[p];
        if (kind != 0) {
            const int dir = s_dir[p];
            const int need = s_rem[p];
            int pos, before, count;
            ds_cross<kDsFine / 32>(need, [&](int fo) {
                return __ldcg(a.dfine + p * kDsFine + ds_ord(fo, kDsFine, dir));
            }, lane, pos, before, count);
            if (pos < 0) {
                take = 0;
            } else if (need - before == count) {
                take = pos + 1;
            } else {
                take = pos;
                part = pos;
                rem = need - before;
                if (kind != 3) {  // one degree: its records in the blocks before this one
                    const int f = ds_ord(pos, kDsFine, dir);
                    for (int b = lane; b < (int)blockIdx.x; b += 32)
                        pre += (int)__ldcg(a.dcntb + (size_t)b * nseg * kDsFine + p * kDsFine + f);
                    for (int o = 16; o > 0; o >>= 1) pre += __shfl_xor_sync(DMOLP_FULL_MASK, pre, o);
                    if (lane == 0 && kind == 2) s_walk1 = 1;  // the warps' counts need a walk of the lists
                }
            }
        }
        if (lane == 0) {
            s_ftake[p] = take;
            s_fpart[p] = part;
            s_frem[p] = rem;
            s_pre[p] = pre;
        }
    }
    __syncthreads();
    // a record of the warp's list: its label, key, fine order position, and whether it is an exact tie
    auto list_rec = [&](int i, int &p, uint64_t &key, int &fo, bool &tie) {
        p = -1;
        key = 0;
        fo = -1;
        tie = false;
        if (i < wl) {
            p = wlist[i];
            key = wkey[i];
            int o;
            bins_of(key, p, o, fo);
            tie = fo == s_fpart[p];
        }
    };
    if (s_walk1) {  // exact ties of multi-degree superbins: this warp's count per label
        for (int i0 = 0; i0 < wl; i0 += 32) {
            int p, fo;
            uint64_t key;
            bool tie;
            list_rec(i0 + lane, p, key, fo, tie);
            tie = tie && s_kind[p] == 2;
            const unsigned m = __match_any_sync(DMOLP_FULL_MASK, tie ? p : -1 - lane);
            if (tie && lane == __ffs(m) - 1) s_wc[wid * nseg + p] += __popc(m);
            __syncwarp();
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < kDsWarps * nseg; i += blockDim.x) {
        const int w = i / nseg, p = i - w * nseg;
        int base = s_pre[p];
        for (int x = 0; x < w; ++x) base += s_wc[x * nseg + p];
        s_wrun[i] = base;
    }
    __syncthreads();
    for (int i0 = 0; i0 < wl; i0 += 32) {
        int p, fo;
        uint64_t key;
        bool tie;
        list_rec(i0 + lane, p, key, fo, tie);
        bool take = p >= 0 && fo < s_ftake[p];
        const unsigned m = __match_any_sync(DMOLP_FULL_MASK, tie ? p : -1 - lane);
        if (tie) take = s_wrun[wid * nseg + p] + __popc(m & below) < s_frem[p];
        __syncwarp();
        if (tie && lane == __ffs(m) - 1) s_wrun[wid * nseg + p] += __popc(m);
        __syncwarp();
        emit_window<1>(a.sp, &take, &key, &p, vmask, te, ws, w_stage, w_scnt);  // all lanes
    }
    // ---- labels with a partial superbin of degree >= 2048: their tail segments ----
    // Every block takes its slice of every such segment's records of fine bins before the partial one.
    for (int p = 0; p < nseg; ++p) {
        if (s_kind[p] != 3) continue;  // block-uniform
        const int nt = __ldcg(a.tcnt + p);
        const int ch = (nt + (int)gridDim.x - 1) / (int)gridDim.x;
        const int lo = (int)blockIdx.x * ch, hi = min(nt, lo + ch);
        const uint64_t *seg_tail = a.tail + s_toff[p];
        const int ftake = s_ftake[p];
        for (int i0 = lo; i0 < hi; i0 += blockDim.x) {  // block-uniform trip count
            const int i = i0 + (int)threadIdx.x;
            bool take = false;
            uint64_t key = 0;
            int pp = p;
            if (i < hi) {
                key = __ldcg(seg_tail + i);
                int o, fo;
                bins_of(key, p, o, fo);
                take = fo < ftake;
            }
            emit_window<1>(a.sp, &take, &key, &pp, vmask, te, ws, w_stage, w_scnt);  // all lanes
        }
    }
    // Block p (p, p + gridDim.x, ...) takes label p's records of the partial fine bin.  It spans 2^jw degrees
    // (octave j, jw = j - 6); its records are counted per sub-bin of the label's order (one degree each while
    // jw <= 10, else 2^(jw-10) degrees), a block scan finds the sub-bin where the rest of the need is reached,
    // the sub-bins before it are taken, and only that sub-bin's records are sorted by key (degree, then id)
    // -- at these degrees usually a handful.
    for (int p = blockIdx.x; p < nseg; p += gridDim.x) {
        if (s_kind[p] != 3) continue;  // block-uniform
        const int nt = __ldcg(a.tcnt + p);
        const uint64_t *seg_tail = a.tail + s_toff[p];
        const int fpart = s_fpart[p], frem = s_frem[p], dir = s_dir[p];
        const int jw = ds_ord(s_opart[p], kDsBins, dir) - kDsCoarse0 + 5;  // superbin kDsCoarse0 + j - 11
        const int sh = jw > 10 ? jw - 10 : 0;
        const int nsub = 1 << (jw - sh);  // <= 1024 = blockDim.x
        auto sub_of = [&](uint64_t key) {
            const int dk = (int)(key >> ibits);
            const int x = (dir ? maxdeg - dk : dk) & ((1 << jw) - 1);
            return (dir ? (1 << jw) - 1 - x : x) >> sh;
        };
        unsigned int *s_sub = reinterpret_cast<unsigned int *>(s_tkey);  // counts first, the tied keys later
        __syncthreads();  // s_ntie and the shared tie keys are free
        for (int i = threadIdx.x; i < nsub; i += blockDim.x) s_sub[i] = 0u;
        if (threadIdx.x == 0) {
            s_ntie = 0;
            s_bstar = -1;
            s_before = 0;
        }
        __syncthreads();
        // pass 1: the partial fine bin's records counted per sub-bin (four keys per thread in flight)
        for (int i0 = 0; i0 < nt; i0 += 4 * blockDim.x) {
            uint64_t k4[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = i0 + q * (int)blockDim.x + (int)threadIdx.x;
                k4[q] = i < nt ? __ldcg(seg_tail + i) : ~0ull;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (k4[q] == ~0ull) continue;
                int o, fo;
                bins_of(k4[q], p, o, fo);
                if (fo == fpart) atomicAdd(&s_sub[sub_of(k4[q])], 1u);
            }
        }
        __syncthreads();
        {  // the sub-bin where the running count reaches frem (block scan, one sub-bin per thread)
            const unsigned int c = (int)threadIdx.x < nsub ? s_sub[threadIdx.x] : 0u;
            unsigned int incl = c;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(DMOLP_FULL_MASK, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) s_wsum[wid] = incl;
            __syncthreads();
            if (wid == 0) {
                unsigned int x = s_wsum[lane];
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned int y = __shfl_up_sync(DMOLP_FULL_MASK, x, o);
                    if (lane >= o) x += y;
                }
                s_wsum[lane] = x;
            }
            __syncthreads();
            incl += wid ? s_wsum[wid - 1] : 0u;
            if (c && incl - c < (unsigned)frem && (unsigned)frem <= incl) {
                s_bstar = (int)threadIdx.x;
                s_before = (int)(incl - c);
            }
        }
        __syncthreads();
        const int bstar = s_bstar, rem2 = frem - s_before;  // bstar < 0: inconsistent counts (never expected)
        // pass 2: sub-bins before bstar are taken, bstar's records collected
        for (int i0 = 0; i0 < nt; i0 += blockDim.x) {
            const int i = i0 + (int)threadIdx.x;
            bool take = false;
            uint64_t key = 0;
            int pp = p;
            if (i < nt && bstar >= 0) {
                key = __ldcg(seg_tail + i);
                int o, fo;
                bins_of(key, p, o, fo);
                if (fo == fpart) {
                    const int sb2 = sub_of(key);
                    if (sb2 < bstar) {
                        take = true;
                    } else if (sb2 == bstar) {
                        const int q = atomicAdd(&s_ntie, 1);
                        if (q < kDsTieCap) s_tkey[q] = key;
                    }
                }
            }
            emit_window<1>(a.sp, &take, &key, &pp, vmask, te, ws, w_stage, w_scnt);  // all lanes
        }
        __syncthreads();
        const int m = s_ntie;
        if (bstar < 0) {
            // nothing more from this label
        } else if (m <= kDsTieCap) {
            // the sub-bin's records sorted by key (bitonic, padded to a power of two): the first rem2 are taken
            int n2 = 1;
            while (n2 < m) n2 <<= 1;
            for (int i = m + (int)threadIdx.x; i < n2; i += blockDim.x) s_tkey[i] = ~0ull;
            for (int size = 2; size <= n2; size <<= 1) {
                for (int stride = size >> 1; stride > 0; stride >>= 1) {
                    __syncthreads();
                    for (int i = threadIdx.x; i < (n2 >> 1); i += blockDim.x) {
                        const int lo = 2 * stride * (i / stride) + (i % stride), hi = lo + stride;
                        const uint64_t x = s_tkey[lo], y = s_tkey[hi];
                        if ((x > y) == ((lo & size) == 0)) {
                            s_tkey[lo] = y;
                            s_tkey[hi] = x;
                        }
                    }
                }
            }
            __syncthreads();
            const int nt2 = rem2 < m ? rem2 : m;
            for (int i0 = 0; i0 < nt2; i0 += blockDim.x) {
                const int i = i0 + (int)threadIdx.x;
                bool take = i < nt2;
                uint64_t key = take ? s_tkey[i] : 0;
                int pp = p;
                emit_window<1>(a.sp, &take, &key, &pp, vmask, te, ws, w_stage, w_scnt);  // all lanes
            }
        } else {  // more ties than the shared keys hold: each ranked against the sub-bin in global memory
            for (int i0 = 0; i0 < nt; i0 += blockDim.x) {
                const int i = i0 + (int)threadIdx.x;
                bool take = false;
                uint64_t key = 0;
                int pp = p;
                if (i < nt) {
                    key = __ldcg(seg_tail + i);
                    int o, fo;
                    bins_of(key, p, o, fo);
                    if (fo == fpart && sub_of(key) == bstar) {
                        int rank = 0;
                        for (int j = 0; j < nt; ++j) {
                            const uint64_t kj = __ldcg(seg_tail + j);
                            int oj, foj;
                            bins_of(kj, p, oj, foj);
                            rank += foj == fpart && sub_of(kj) == bstar && kj < key;
                        }
                        take = rank < rem2;
                    }
                }
                emit_window<1>(a.sp, &take, &key, &pp, vmask, te, ws, w_stage, w_scnt);  // all lanes
            }
        }
    }
    // ---- end: the warps' staged appends and the block's sums, one atomic per list and per sum for the block
    //      (one per warp would queue ~4,700 atomics on each of six counters) ----
    __syncthreads();  // every warp's stage and counts are final
    if (threadIdx.x < 4) {
        const int j = threadIdx.x;
        int tot = 0;
        for (int w = 0; w < kDsWarps; ++w) {
            s_soff[w][j] = tot;
            tot += s_scnt[w][j];
        }
        s_sbase[j] = tot ? atomicAdd(list_ctr(a.sp, j), tot) : 0;
    }
    te = warp_sum_u64(te);
    ws = warp_sum_u64(ws);
    if (lane == 0) {
        s_te[wid] = te;
        s_ws[wid] = ws;
    }
    __syncthreads();
    for (int j = 0; j < 4; ++j) {
        const int n = w_scnt[j];
        int *dst = list_ptr(a.sp, j) + s_sbase[j] + s_soff[wid][j];
        for (int i = lane; i < n; i += 32) dst[i] = w_stage[j * kStage + i];
    }
    if (threadIdx.x == 0) {
        unsigned long long tt = 0, ww = 0;
        for (int w = 0; w < kDsWarps; ++w) {
            tt += s_te[w];
            ww += s_ws[w];
        }
        if (tt) atomicAdd(a.sp.te, tt);
        if (ww) atomicAdd(a.sp.wsum, ww);
    }
}

}  // namespace

void select_window(dmolp_ctx *c, int nseg, int keybits, const SplitArgs &split, const int *stopped,
                   bool first_hist_ready) {
    SelArgs a = select_args(c, nseg, keybits);
    a.n_dev = &c->b.cnt->npos;
    a.stopped = stopped;
    a.sp = split;
    a.hist_ready = first_hist_ready ? 1 : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c->num_sms);  // one block per SM, all resident (cooperative launch)
    cfg.blockDim = dim3(kSelThreads);
    cfg.dynamicSmemBytes = select_smem_bytes(nseg);
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_select, a);
    if (e != cudaSuccess && c->launch_error == cudaSuccess) c->launch_error = e;  // reported by the entry point
    c->launches += 1;
}

bool select_window_deg(dmolp_ctx *c, int nseg, const SplitArgs &split, const int *stopped) {
    if (nseg > kDegSelMaxK) return false;
    DegSelArgs a;
    a.seg = c->b.bown;
    a.key = c->b.bkey;
    a.n_dev = &c->b.cnt->npos;
    a.lists = c->b.active[0];
    a.lkeys = c->b.dlkey;
    a.tail = c->b.dtkey;
    a.tcnt = c->b.dtcnt + (split.t & 1) * kDegSelMaxK;
    a.tcnt_next = c->b.dtcnt + ((split.t + 1) & 1) * kDegSelMaxK;
    a.dsup = c->b.dsup;
    a.dfine = c->b.dfine[split.t & 1];
    a.dfine_next = c->b.dfine[(split.t + 1) & 1];
    a.dcntb = c->b.dcntb;
    a.nseg = nseg;
    a.polls = c->wait_polls;
    a.ctl = c->b.ctrl;
    a.stopped = stopped;
    a.sp = split;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c->num_sms);  // one block per SM, all resident (cooperative launch)
    cfg.blockDim = dim3(kDsThreads);
    cfg.dynamicSmemBytes = ds_smem_bytes(nseg);
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_select_deg, a);
    if (e != cudaSuccess && c->launch_error == cudaSuccess) c->launch_error = e;  // reported by the entry point
    c->launches += 1;
    return true;
}

int select_binary_version() {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k_select) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return fa.binaryVersion;
}

void select_prepare() {
    cudaFuncSetAttribute(k_select_deg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ds_smem_bytes(kDegSelMaxK));
    cudaFuncSetAttribute(k_select, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)select_smem_bytes(kSmemSegMax));
    p1_prepare();
    loop_prepare();
}

}  // namespace dmolp
