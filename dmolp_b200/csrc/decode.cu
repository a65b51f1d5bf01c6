// Decoder of the learned proposal: recursive inertial bisection of the proposal coordinates P (8 wide) of a
// graph's vertices into k balanced labels, a team of CTAs per graph (team.cuh).
//
// Every part with kp >= 2 labels splits (all parts of a level at once) into kl = kp/2 and kp - kl labels; the
// left child takes the floor(n * kl / kp) vertices with the smallest (projection, id) on the part's principal
// axis.  The axis: mean and covariance of the part in double, cyclic Jacobi on the 8x8 covariance, the
// eigenvector of the largest eigenvalue signed so that its largest-magnitude component is positive.
//
// A part's vertices stay contiguous in a permutation (ascending ids), so each warp owns a run of it.  For the sums the
// parts are cut into segments whose length the graph and the level alone decide (segment_length).  A warp sums a segment
// at a time in registers, to the segment's record in global memory, and one warp per part adds the records in order.
// So the sums' order, and with it the result, depends neither
// on scheduling nor on the team, that is on what else is in the batch.  (Sums over whatever vertices a warp held did:
// the team's size moved the last bits of mean and axis.)  The selection is an MSD radix select over keys (orderable
// float bits of the projection, id) with 6-bit digits and no lists: a record is open while its leading digits are its
// part's prefix.  A stable partition of the permutation by the part's threshold key then forms the children.
//
// What bounds it: passes over 32 bytes per vertex at the level's start, and the chain of about 20 barriers per
// level.  One CTA that walked all vertices once per part took 229 ms for a skewed graph of a million vertices and
// 32 parts; 16 CTAs over the permutation take 2.7 ms.
#include <algorithm>
#include <vector>

#include "mpnn.cuh"
#include "team.cuh"

namespace dmolp {
namespace mpnn {
namespace {

using batch::ClusterTeam;
using batch::CtaTeam;
using batch::kDigitBits;
using batch::kDigits;

constexpr int kDecThreads = 512;
constexpr int kWarps = kDecThreads / 32;
constexpr int kParts = batch::kBatchMaxK;
constexpr int kDims = 8;
constexpr int kTri = kDims * (kDims + 1) / 2;
constexpr int kRun = 128;             // granularity of the warps' runs, in vertices; the shortest segment
constexpr int kRecs = kWarps + kParts;  // a CTA's warps meet at most this many (warp, part) pairs
static_assert(kRun == kDecSeg && kTri == kDecRecord && kParts / 2 == kDecSplits, "the records' workspace");

// Vertices per segment where `split` parts of n vertices together split.  For t segments per warp of the largest team
// the length is the shortest that leaves at most so many (a part's last segment may be short); t is chosen by the
// level's time, t x (length / 32 + kReduce), in steps of 32 vertices: a segment's sums over the lanes cost about
// kReduce of them.  So a large graph takes one or two segments per warp at every level, a small one segments of kRun.
// (Lengths of 512 and more by the part's size: a graph of 28 K vertices left three of four warps without a segment of
// the first part, its decoder 0.53 -> 0.58 ms; one length per graph: 2.76 -> 3.07 ms for a million vertices.)
constexpr int kReduce = 6;
__device__ __forceinline__ int segment_length(int n, int split) {
    int best = 0x7fffffff, len = kRun;
    for (int t = 1; t <= 4; ++t) {
        const int m = t * kWarps * batch::kMaxTeam - split;
        const int steps = ((n - 1) / m + 32) / 32, cost = t * (steps + kReduce);
        if (cost < best) {
            best = cost;
            len = steps * 32;
        }
    }
    return len < kRun ? kRun : len;
}

struct DecSmem {
    double mean[kParts][kDims], axis[kParts][kDims];
    double A[kWarps][kDims][kDims], V[kWarps][kDims][kDims];  // eigen-decomposition, a matrix per warp
    uint64_t prefix[kParts], cut[kParts];  // selection: digits fixed so far; keys below cut are selected
    int hist[2][kParts * kDigits];         // zero between selections
    int lrec[kRecs];                       // selected vertices per (warp, part)
    int kp[kParts], beg[kParts], cnt[kParts], need[kParts], below[kParts], keep[kParts], fin[kParts];
    int part[kParts], run0[kParts + 1], seg0[kParts + 1];  // splitting parts by ordinal, their first runs and segments
    int len, nsplit, bad, inst;  // len: vertices per segment
};

__device__ __forceinline__ unsigned orderable(float x) {
    const unsigned u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Eigen-decomposition of a symmetric 8x8 matrix by one warp (cyclic Jacobi, double; lane r < 8 holds row or
// column r of each rotation); eigenvalues on the diagonal of A, eigenvectors in the columns of V.
__device__ void jacobi8(double (*A)[kDims], double (*V)[kDims]) {
    const int r = threadIdx.x & 31;
    const bool on = r < kDims;
    if (on)
        for (int j = 0; j < kDims; ++j) V[r][j] = r == j ? 1.0 : 0.0;
    __syncwarp();
    for (int sweep = 0; sweep < 50; ++sweep) {
        double off = 0.0;
        for (int p = 0; p < kDims; ++p)
            for (int q = p + 1; q < kDims; ++q) off += A[p][q] * A[p][q];
        if (off < 1e-30) break;
        for (int p = 0; p < kDims; ++p)
            for (int q = p + 1; q < kDims; ++q) {
                const double apq = A[p][q];
                if (fabs(apq) < 1e-300) continue;
                const double theta = (A[q][q] - A[p][p]) / (2.0 * apq);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
                __syncwarp();
                if (on) {
                    const double arp = A[r][p], arq = A[r][q];
                    A[r][p] = c * arp - sn * arq;
                    A[r][q] = sn * arp + c * arq;
                }
                __syncwarp();
                if (on) {
                    const double apr = A[p][r], aqr = A[q][r];
                    A[p][r] = c * apr - sn * aqr;
                    A[q][r] = sn * apr + c * aqr;
                    const double vrp = V[r][p], vrq = V[r][q];
                    V[r][p] = c * vrp - sn * vrq;
                    V[r][q] = sn * vrp + c * vrq;
                }
                __syncwarp();
            }
    }
    __syncwarp();
}

// A warp's share of a level: the runs [a, b) of the splitting parts, whose runs follow each other by ordinal.
// f(ordinal, first position, last position) for each part it meets, positions in the permutation.
template <typename F>
__device__ __forceinline__ void for_parts(const DecSmem &sm, int a, int b, F f) {
    int o = 0;
    while (o < sm.nsplit && sm.run0[o + 1] <= a) ++o;
    for (; a < b; ++o) {
        const int p = sm.part[o], r0 = sm.run0[o];
        const int z = b < sm.run0[o + 1] ? b : sm.run0[o + 1];
        const int i0 = sm.beg[p] + (a - r0) * kRun;
        const int i1 = z == sm.run0[o + 1] ? sm.beg[p] + sm.cnt[p] : sm.beg[p] + (z - r0) * kRun;
        f(o, i0, i1);
        a = z;
    }
}

// The segments [a, b) one by one, numbered alike: f(ordinal, segment, first position, last position).
template <typename F>
__device__ __forceinline__ void for_segments(const DecSmem &sm, int a, int b, F f) {
    int o = 0;
    for (; a < b; ++a) {
        while (sm.seg0[o + 1] <= a) ++o;
        const int p = sm.part[o], end = sm.beg[p] + sm.cnt[p];
        const int i0 = sm.beg[p] + (a - sm.seg0[o]) * sm.len;
        f(o, a, i0, end - i0 < sm.len ? end : i0 + sm.len);
    }
}

// Sums over the warp's lanes of N values each (a power of two): lane l returns the sum of x[l % N].  Halves of the
// values are exchanged, so N - 1 shuffles do what 5 N would; the tree of additions is that of the butterfly.
template <int N>
__device__ __forceinline__ double lane_sums(double *x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = N / 2; w > 0; w >>= 1) {
        const bool up = lane & w;
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const double give = up ? x[i] : x[i + w], keep = up ? x[i + w] : x[i];
            x[i] = keep + __shfl_xor_sync(DMOLP_FULL_MASK, give, w);
        }
    }
#pragma unroll
    for (int o = N; o < 32; o <<= 1) x[0] += __shfl_xor_sync(DMOLP_FULL_MASK, x[0], o);
    return x[0];
}

// The sums of the records of the segments [s, e), of width n <= kTri, in order, to lanes: lane l returns entries l and
// l + 32.  Written by other CTAs: read past L1.
__device__ __forceinline__ double2 add_records(const double *rec, int s, int e, int n) {
    const int lane = threadIdx.x & 31;
    double2 t = make_double2(0.0, 0.0);
    for (; s < e; s += 8) {  // eight records in flight
        double x[8], y[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double *r = rec + (size_t)(s + q) * kTri + lane;
            x[q] = s + q < e && lane < n ? __ldcg(r) : 0.0;
            y[q] = s + q < e && lane + 32 < n ? __ldcg(r + 32) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            t.x += x[q];
            t.y += y[q];
        }
    }
    return t;
}

template <typename Tm>
__device__ void run_decode(const DecodeWork &w, int ii, const Tm &tm, DecSmem &sm) {
    const batch::Inst I = w.inst[ii];
    const int k = I.k, nv = I.nv, vb = (int)I.vbase;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int team_warps = tm.threads() / 32;
    const int wid = tm.rank_of() * kWarps + wib;  // a CTA's warps are consecutive here
    int32_t *perm[2] = {w.l0 + vb, w.l1 + vb};
    uint64_t *const key = w.key + vb;  // by position in the permutation
    double *const rec = w.rec + decode_record(vb, ii) * kTri;
    const float *const Z = w.Z + (size_t)vb * 16;
    const int bits = 32 + I.ibits, npass = (bits + kDigitBits - 1) / kDigitBits, top = npass * kDigitBits;
    auto coords = [&](int v, float (&x)[kDims]) {
        const float4 *z = reinterpret_cast<const float4 *>(Z + (size_t)v * 16);
        const float4 z0 = z[0], z1 = z[1];
        x[0] = z0.x; x[1] = z0.y; x[2] = z0.z; x[3] = z0.w;
        x[4] = z1.x; x[5] = z1.y; x[6] = z1.z; x[7] = z1.w;
    };

    if (threadIdx.x == 0) sm.bad = 0;
    for (int p = threadIdx.x; p < kParts; p += kDecThreads) {
        sm.kp[p] = p == 0 ? k : 0;
        sm.beg[p] = 0;
        sm.cnt[p] = p == 0 ? nv : 0;
    }
    for (int i = threadIdx.x; i < 2 * kParts * kDigits; i += kDecThreads) (&sm.hist[0][0])[i] = 0;
    tm.sync();
    for (int v = tm.thread(); v < nv; v += tm.threads()) {
        w.label[vb + v] = 0;
        perm[0][v] = v;
        float x[kDims];
        coords(v, x);
        bool ok = true;
#pragma unroll
        for (int d = 0; d < kDims; ++d) ok &= isfinite(x[d]);
        if (!ok) *tm.first(&sm.bad) = 1;
    }
    tm.sync();
    if (*tm.first(&sm.bad) || nv < k) {  // not usable: the caller falls back
        if (tm.is_first() && threadIdx.x == 0) w.status[ii] = 1;
        tm.sync();
        return;
    }
    int cur = 0;
    for (int level = 0; level < 7; ++level, cur ^= 1) {
        // ---- the splitting parts, their runs and segments (by every CTA alike) ----
        __syncthreads();
        if (wib == 0) {
            int nsplit = 0, total = 0, runs = 0, segs = 0;
            for (int p0 = 0; p0 < kParts; p0 += 32) {
                const int n = sm.kp[p0 + lane] >= 2 ? sm.cnt[p0 + lane] : 0;
                nsplit += __popc(__ballot_sync(DMOLP_FULL_MASK, n > 0));
                total += __reduce_add_sync(DMOLP_FULL_MASK, n);
            }
            const int len = segment_length(total, nsplit);
            nsplit = 0;
            for (int p0 = 0; p0 < kParts; p0 += 32) {
                const int p = p0 + lane;
                const bool split = sm.kp[p] >= 2 && sm.cnt[p] > 0;
                const int r = split ? (sm.cnt[p] - 1) / kRun + 1 : 0, g = split ? (sm.cnt[p] - 1) / len + 1 : 0;
                int ir = r, ig = g;
                for (int o = 1; o < 32; o <<= 1) {
                    const int yr = __shfl_up_sync(DMOLP_FULL_MASK, ir, o), yg = __shfl_up_sync(DMOLP_FULL_MASK, ig, o);
                    if (lane >= o) {
                        ir += yr;
                        ig += yg;
                    }
                }
                const unsigned m = __ballot_sync(DMOLP_FULL_MASK, split);
                if (split) {
                    const int o = nsplit + __popc(m & ((1u << lane) - 1));
                    sm.part[o] = p;
                    sm.run0[o] = runs + ir - r;
                    sm.seg0[o] = segs + ig - g;
                }
                nsplit += __popc(m);
                runs += __shfl_sync(DMOLP_FULL_MASK, ir, 31);
                segs += __shfl_sync(DMOLP_FULL_MASK, ig, 31);
            }
            if (lane == 0) {
                sm.nsplit = nsplit;
                sm.run0[nsplit] = runs;
                sm.seg0[nsplit] = segs;
                sm.len = len;
            }
        }
        for (int p = threadIdx.x; p < kParts; p += kDecThreads) {
            const bool split = sm.kp[p] >= 2 && sm.cnt[p] > 0;
            sm.need[p] = split ? (int)(((long long)sm.cnt[p] * (sm.kp[p] / 2)) / sm.kp[p]) : 0;
            sm.prefix[p] = 0;
            sm.fin[p] = !split;
        }
        bool any = false;
        for (int p = lane; p < kParts; p += 32) any |= sm.kp[p] >= 2;
        any = __any_sync(DMOLP_FULL_MASK, any);
        __syncthreads();
        if (!any) break;
        const int nsplit = sm.nsplit, runs = sm.run0[nsplit], segs = sm.seg0[nsplit];
        const int per = runs > 0 ? (runs + team_warps - 1) / team_warps : 1;
        const int a = min(wid * per, runs), b = min(a + per, runs);
        const int sper = (segs + team_warps - 1) / team_warps;
        const int sa = min(wid * sper, segs), sb = min(sa + sper, segs);
        const int32_t *const pm = perm[cur];
        // ---- means ----
        for_segments(sm, sa, sb, [&](int, int seg, int i0, int i1) {
            double acc[kDims];
#pragma unroll
            for (int d = 0; d < kDims; ++d) acc[d] = 0.0;
            for (int i = i0 + lane; i < i1; i += 32) {
                float x[kDims];
                coords(pm[i], x);
#pragma unroll
                for (int d = 0; d < kDims; ++d) acc[d] += (double)x[d];
            }
            const double t = lane_sums<kDims>(acc);
            if (lane < kDims) rec[(size_t)seg * kTri + lane] = t;
        });
        tm.sync();
        for (int o = tm.warp(); o < nsplit; o += team_warps) {
            const double s = add_records(rec, sm.seg0[o], sm.seg0[o + 1], kDims).x / (double)sm.cnt[sm.part[o]];
            if (lane < kDims)
                for (int r = 0; r < tm.size(); ++r) *tm.at(&sm.mean[o][lane], r) = s;
        }
        tm.sync();
        // ---- covariances (upper triangles), principal axes ----
        for_segments(sm, sa, sb, [&](int o, int seg, int i0, int i1) {
            double acc[kTri], mu[kDims];
#pragma unroll
            for (int i = 0; i < kTri; ++i) acc[i] = 0.0;
#pragma unroll
            for (int d = 0; d < kDims; ++d) mu[d] = sm.mean[o][d];
            for (int i = i0 + lane; i < i1; i += 32) {
                float xf[kDims];
                coords(pm[i], xf);
                double x[kDims];
#pragma unroll
                for (int d = 0; d < kDims; ++d) x[d] = (double)xf[d] - mu[d];
                int q = 0;
#pragma unroll
                for (int c = 0; c < kDims; ++c)
#pragma unroll
                    for (int e = c; e < kDims; ++e) acc[q++] += x[c] * x[e];
            }
            const double t0 = lane_sums<32>(acc), t1 = lane_sums<kTri - 32>(acc + 32);
            rec[(size_t)seg * kTri + lane] = t0;
            if (lane < kTri - 32) rec[(size_t)seg * kTri + 32 + lane] = t1;
        });
        tm.sync();
        for (int o = tm.warp(); o < nsplit; o += team_warps) {
            const double2 s = add_records(rec, sm.seg0[o], sm.seg0[o + 1], kTri);
            double(*A)[kDims] = sm.A[wib], (*V)[kDims] = sm.V[wib];
            int q = 0;
            for (int c = 0; c < kDims; ++c)
                for (int e = c; e < kDims; ++e, ++q)
                    if (lane == (q & 31)) A[c][e] = A[e][c] = q < 32 ? s.x : s.y;
            __syncwarp();
            jacobi8(A, V);
            int bi = 0;  // largest eigenvalue, lowest index on ties
            for (int r = 1; r < kDims; ++r)
                if (A[r][r] > A[bi][bi]) bi = r;
            int mi = 0;
            for (int r = 1; r < kDims; ++r)
                if (fabs(V[r][bi]) > fabs(V[mi][bi])) mi = r;
            const double sg = V[mi][bi] < 0 ? -1.0 : 1.0;
            if (lane < kDims)
                for (int r = 0; r < tm.size(); ++r) *tm.at(&sm.axis[o][lane], r) = sg * V[lane][bi];
            __syncwarp();
        }
        tm.sync();
        // ---- projections: keys by position, first digit ----
        for_parts(sm, a, b, [&](int o, int i0, int i1) {
            const int p = sm.part[o];
            double mu[kDims], ax[kDims];
#pragma unroll
            for (int d = 0; d < kDims; ++d) {
                mu[d] = sm.mean[o][d];
                ax[d] = sm.axis[o][d];
            }
            for (int i = i0 + lane; i < i1; i += 32) {
                const int v = pm[i];
                float x[kDims];
                coords(v, x);
                double y = 0.0;
#pragma unroll
                for (int d = 0; d < kDims; ++d) y += ((double)x[d] - mu[d]) * ax[d];
                const uint64_t kx = ((uint64_t)orderable((float)y) << I.ibits) | (uint64_t)v;
                key[i] = kx;
                atomicAdd(&sm.hist[0][p * kDigits + (int)((kx >> (top - kDigitBits)) & (kDigits - 1))], 1);
            }
        });
        tm.sync();
        // ---- per splitting part the threshold under which its need smallest keys lie ----
        for (int pass = 0; pass < npass; ++pass) {
            const int shift = top - kDigitBits * (pass + 1);
            batch::cut_digit(tm, kParts, sm.hist[pass & 1], sm.need, sm.below, sm.keep);
            tm.sync();
            for (int p = threadIdx.x; p < kParts; p += kDecThreads) {
                if (sm.fin[p]) continue;
                if (sm.keep[p] < 0) {
                    sm.fin[p] = 1;
                    sm.cut[p] = ((sm.prefix[p] << kDigitBits) + (uint64_t)sm.below[p]) << shift;
                } else {
                    sm.prefix[p] = (sm.prefix[p] << kDigitBits) | (uint64_t)sm.keep[p];
                }
            }
            for (int i = threadIdx.x; i < kParts * kDigits; i += kDecThreads) sm.hist[pass & 1][i] = 0;
            const bool open = batch::any_open(kParts, sm.keep);
            __syncthreads();
            if (!open) break;
            for_parts(sm, a, b, [&](int o, int i0, int i1) {
                const int p = sm.part[o];
                if (sm.fin[p]) return;
                const uint64_t pre = sm.prefix[p];
                int *const h = sm.hist[(pass + 1) & 1] + p * kDigits;
                for (int i = i0 + lane; i < i1; i += 32) {
                    const uint64_t kx = key[i];
                    if ((kx >> shift) == pre) atomicAdd(&h[(int)((kx >> (shift - kDigitBits)) & (kDigits - 1))], 1);
                }
            });
            tm.sync();
        }
        // ---- children: a stable partition of each part's positions by its threshold ----
        for_parts(sm, a, b, [&](int o, int i0, int i1) {
            const uint64_t cut = sm.cut[sm.part[o]];
            int n = 0;
            for (int i = i0 + lane; i < i1; i += 32) n += key[i] < cut;
            n = __reduce_add_sync(DMOLP_FULL_MASK, n);
            if (lane == 0) sm.lrec[wib + o] = n;
        });
        tm.sync();
        for_parts(sm, a, b, [&](int o, int i0, int i1) {
            const int p = sm.part[o], kl = sm.kp[p] / 2, kr = sm.kp[p] - kl;
            const uint64_t cut = sm.cut[p];
            // selected vertices of the part in front of this share: its earlier warps' counts
            int left = 0;
            for (int x = sm.run0[o] / per + lane; x < wid; x += 32)
                left += *tm.at(&sm.lrec[x % kWarps + o], x / kWarps);
            left = __reduce_add_sync(DMOLP_FULL_MASK, left);
            const int nl = (int)(((long long)sm.cnt[p] * kl) / sm.kp[p]);
            for (int j0 = i0; j0 < i1; j0 += 32) {
                const int i = j0 + lane;
                const bool in = i < i1, sel = in && key[i] < cut;
                const unsigned m = __ballot_sync(DMOLP_FULL_MASK, sel);
                if (in) {
                    const int v = pm[i], before = left + __popc(m & ((1u << lane) - 1));
                    const int at = sel ? before : nl + (i - sm.beg[p]) - before;
                    perm[cur ^ 1][sm.beg[p] + at] = v;
                    if ((sel ? kl : kr) == 1) w.label[vb + v] = sel ? p : p + kl;  // the part is final
                }
                left += __popc(m);
            }
        });
        tm.sync();  // counts and tables are read before they change; the new order is complete
        if (wib == 0) {  // a child p + kl never falls on a part that still splits: its labels are [p, p + kp)
            int kp[2], beg[2], cnt[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                kp[q] = sm.kp[lane + 32 * q];
                beg[q] = sm.beg[lane + 32 * q];
                cnt[q] = sm.cnt[lane + 32 * q];
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int p = lane + 32 * q;
                if (kp[q] < 2) continue;
                const int kl = kp[q] / 2, nl = (int)(((long long)cnt[q] * kl) / kp[q]);
                sm.kp[p] = kl;
                sm.cnt[p] = nl;
                sm.kp[p + kl] = kp[q] - kl;
                sm.beg[p + kl] = beg[q] + nl;
                sm.cnt[p + kl] = cnt[q] - nl;
            }
        }
    }
    // ---- usable only if no part ended empty ----
    if (tm.is_first()) {
        bool empty = false;
        for (int p = threadIdx.x; p < k; p += kDecThreads) empty |= sm.cnt[p] == 0;
        empty = __syncthreads_or(empty);
        if (threadIdx.x == 0) w.status[ii] = empty ? 1 : 0;
    }
    tm.sync();  // no CTA leaves, or starts on another graph, while its tables are read
}

__global__ void __launch_bounds__(kDecThreads, 1) k_decode(DecodeWork w, const int32_t *order, int n) {
    extern __shared__ __align__(16) unsigned char dyn[];
    DecSmem &sm = *reinterpret_cast<DecSmem *>(dyn);
    const CtaTeam<kDecThreads> tm;
    for (;;) {
        if (threadIdx.x == 0) sm.inst = atomicAdd(w.next, 1);
        __syncthreads();
        const int q = sm.inst;
        __syncthreads();
        if (q >= n) break;
        run_decode(w, order[q], tm, sm);
    }
}

__global__ void __launch_bounds__(kDecThreads, 1) k_decode_team(DecodeWork w, const int32_t *order) {
    extern __shared__ __align__(16) unsigned char dyn[];
    const ClusterTeam<kDecThreads> tm;
    run_decode(w, order[blockIdx.x / tm.size()], tm, *reinterpret_cast<DecSmem *>(dyn));
}

int decode_max_team() {
    for (int c = batch::kMaxTeam; c > 1; c >>= 1) {
        int n = 0;
        if (batch::max_clusters(k_decode_team, c, kDecThreads, &n, sizeof(DecSmem)) && n > 0) return c;
    }
    return 1;
}

}  // namespace

int decode(const DecodeWork &w, const std::vector<int32_t> &order, const int32_t *d_order, const batch::View &b,
           cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(k_decode, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_decode_team, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecSmem));
    if (e != cudaSuccess) return (int)e;
    const batch::TeamPlan plan = batch::team_sizes(*b.h_inst, order, b.num_sms, kDecThreads, decode_max_team());
    cudaMemsetAsync(w.next, 0, sizeof(int), s);
    b.fork->open(plan, s);
    for (int j = 0, c = batch::kMaxTeam; c > 1; ++j, c >>= 1) {
        if (plan.n[j] > 0)
            batch::launch_cluster_smem(k_decode_team, plan.n[j], c, kDecThreads, sizeof(DecSmem),
                                       b.fork->stream(plan, j, s), w, d_order);
        d_order += plan.n[j];
    }
    const int j1 = batch::kTeamClasses - 1, n1 = plan.n[j1];
    if (n1 > 0)
        k_decode<<<std::min(b.num_sms, n1), kDecThreads, sizeof(DecSmem), b.fork->stream(plan, j1, s)>>>(w, d_order, n1);
    b.fork->close(plan, s);
    return (int)cudaGetLastError();
}

}  // namespace mpnn
}  // namespace dmolp
