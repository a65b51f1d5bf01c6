// Learned initial-partition proposal: the kernels of a 3-layer mean-aggregation message-passing network
// (BF16 weights and activations, FP32 accumulation on the tcgen05 tensor cores) and its training step.  Its
// input features are in features.cu, the decoder of its embedding in decode.cu.
//
//   layer l:  Z_l = [H_l | mean over neighbours of H_l] @ W_l + b_l,   H_{l+1} = ReLU(Z_l)  (l = 1, 2)
//   sizes:    16 -> 64 -> 64 -> 16;  inputs: degree / mean degree, log(1 + degree), 8 random-walk
//             features, k / 64 (the remaining input columns are 0)
//
// The concatenation [H | mean H] is one BF16 buffer per layer: the GEMM epilogue of layer l writes H_{l+1}
// into the left half of layer l+1's buffer and the aggregation kernel fills its right half.  The GEMMs
// copy 128-row tiles of A and the whole of B into shared memory in the no-swizzle K-major core-matrix layout
// (umma.cuh), one thread issues tcgen05.mma into a tensor-memory accumulator, completion is signalled on an
// mbarrier (bounded wait: a stuck MMA sets an error flag instead of hanging), and the epilogue reads the
// accumulator with tcgen05.ld.  The weight gradient has the vertices as its reduction axis: both operands are
// MN-major, and each CTA adds its partial sums to dW with atomics.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "mpnn.cuh"
#include "umma.cuh"

namespace dmolp {
namespace mpnn {
namespace {

// Polls of the MMA completion barrier after a GEMM gave up (GemmArgs::polls): the MMA in flight still
// completes before its TMEM is freed; far above any real MMA's time.
constexpr uint32_t kWaitLimit = 1u << 24;

__device__ __forceinline__ uint4 zero4() { return make_uint4(0, 0, 0, 0); }

// 1 / deg as a float (features.cu: the float division is exact to the last bit of the double one).
__device__ __forceinline__ float inv_degree(int64_t deg) {
    if (deg <= 0) return 0.f;
    return deg <= (int64_t(1) << 24) ? __fdiv_rn(1.f, (float)deg) : (float)(1.0 / (double)deg);
}

// ------------------------------------------------------------------------------------------------ GEMM
// What bounds these: bytes.  K is at most 128, so a row's 32 to 256 bytes are read once for at most 16 KFLOP.  The
// row kernels therefore keep the whole weight tile in shared memory, and copy a CTA's next row tile (asynchronously,
// 16 bytes per thread) while the tensor core and the epilogue work on the current one; the weight gradient copies
// its next 64 vertices behind the current MMAs, in the MN-major layout, which takes rows as they are.  Eight
// consecutive threads fill one core matrix: no bank conflicts, and whole sectors of four rows' neighbouring chunks.
// Before, tiles of K = 64 were staged through registers (transposed element by element for the weight gradient) with
// nothing else in flight.  A training step of 64 graphs (0.72 M vertices): its eight GEMMs 1.42 -> 0.63 ms.
constexpr int kGemmThreads = 128;

// Accumulator columns c0 .. c0 + 15 of a warp's 32 rows from row0 on to the outputs, lane r holding row r (inv: its
// 1 / degree for the data gradient).  They go through the warp's shared stage, so that neighbouring lanes write
// neighbouring words: a store of 16 bytes per row took a transaction per lane (128 columns out of K = 16: 167 us for
// 0.72 M rows, now 101).
constexpr int kStagePitch = 20;  // floats per row: 16-byte aligned, conflict-free by rows
constexpr size_t kStageBytes = (size_t)kGemmThreads * kStagePitch * sizeof(float);

__device__ __forceinline__ void store_rows(const GemmArgs &g, float *stage, int row0, int c0, float inv, float (&v)[16]) {
    const int lane = threadIdx.x & 31;
    if (g.off && c0 >= kHidden) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __fmul_rn(v[i], inv);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if (g.bias) v[i] = __fadd_rn(v[i], g.bias[c0 + i]);
        if (g.relu) v[i] = fmaxf(v[i], 0.0f);
    }
    float4 *mine = reinterpret_cast<float4 *>(stage + lane * kStagePitch);
#pragma unroll
    for (int i = 0; i < 4; ++i) mine[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    __syncwarp();
    if (g.out_bf16) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {  // two lanes per row
            const int r = i * 16 + (lane >> 1), row = row0 + r;
            const float4 *src = reinterpret_cast<const float4 *>(stage + r * kStagePitch) + (lane & 1) * 2;
            const float4 x = src[0], y = src[1];
            const float f[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
            __align__(16) __nv_bfloat16 h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) h[j] = __float2bfloat16_rn(f[j]);
            if (row < g.rows)
                *reinterpret_cast<uint4 *>(g.out_bf16 + (size_t)row * g.ldo + c0 + (lane & 1) * 8) =
                    *reinterpret_cast<const uint4 *>(h);
        }
    }
    if (g.out_f32) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // four lanes per row
            const int r = i * 8 + (lane >> 2), row = row0 + r;
            const float4 x = *(reinterpret_cast<const float4 *>(stage + r * kStagePitch) + (lane & 3));
            if (row < g.rows) *reinterpret_cast<float4 *>(g.out_f32 + (size_t)row * g.ldo32 + c0 + (lane & 3) * 4) = x;
        }
    }
    __syncwarp();  // the stage may be written again
}

// Tensor memory and the completion barrier of a CTA; returns the accumulator's address.
__device__ __forceinline__ uint32_t gemm_begin(uint64_t *mbar, uint32_t *tslot, uint32_t ncol) {
    if (threadIdx.x < 32) umma::tmem_alloc(tslot, ncol);
    if (threadIdx.x == 0) {
        umma::mbar_init(mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    return *tslot;
}

// Nothing is in flight when the CTA ends: copies, MMAs (a wait that gave up is waited for once more), tensor memory.
__device__ __forceinline__ void gemm_end(const GemmArgs &g, bool ok, uint64_t *mbar, uint32_t phase, uint32_t tmem,
                                         uint32_t ncol) {
    umma::copy_wait<0>();
    if (!ok) {
        umma::mbar_wait(mbar, phase, kWaitLimit);  // let an MMA still in flight finish before the free
        if (threadIdx.x == 0) atomicExch(g.err, 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) umma::tmem_free(tmem, ncol);
}

// Rows of A [rows x K] times B^T [N x K]: 128 rows per item.
template <int N, int K>
struct RowGemm {
    static constexpr size_t kTileA = 128 * K * 2, kTileB = (size_t)N * K * 2, kSmem = 2 * kTileA + kTileB + kStageBytes;
    static constexpr uint32_t kCols = N < 32 ? 32 : N;
    // resident CTAs per SM: shared memory, tensor memory (512 columns), and no more than eight
    static constexpr int kFit = (int)(220 * 1024 / (kSmem + 1024)), kTm = 512 / (int)kCols;
    static constexpr int kPerSm = kFit < kTm ? (kFit < 8 ? kFit : 8) : (kTm < 8 ? kTm : 8);
};

template <int N, int K>
__global__ void __launch_bounds__(kGemmThreads) k_gemm_rows(GemmArgs g) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tslot;
    constexpr int CH = K / 8;  // 16-byte chunks per row
    constexpr uint32_t TA = RowGemm<N, K>::kTileA, NCOL = RowGemm<N, K>::kCols;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t tmem = gemm_begin(&mbar, &tslot, NCOL);
    constexpr uint32_t idesc = umma::idesc_bf16_f32(128, N);
    const uint32_t sA = umma::smem_addr(smem), sB = sA + 2 * TA;
    float *const stage =
        reinterpret_cast<float *>(smem + 2 * TA + RowGemm<N, K>::kTileB) + warp * 32 * kStagePitch;
    const int nitems = (g.rows + 127) / 128;
    // chunk q of a tile is row 8 (q / 8 / CH) + q % 8, chunk (q / 8) % CH, and lies at byte 16 q
    for (int q = tid; q < N * CH; q += kGemmThreads) {
        const int n = q / (8 * CH) * 8 + (q & 7), c = (q >> 3) % CH;
        umma::copy16(sB + 16 * q, g.B + (size_t)(n < g.nb ? n : 0) * g.ldb + c * 8, n < g.nb);
    }
    auto load = [&](int item, uint32_t dst) {
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const int q = i * kGemmThreads + tid;
            const int row = item * 128 + q / (8 * CH) * 8 + (q & 7), c = (q >> 3) % CH;
            umma::copy16(dst + 16 * q, g.A + (size_t)min(row, g.rows - 1) * g.lda + c * 8, row < g.rows);
        }
    };
    if ((int)blockIdx.x < nitems) load(blockIdx.x, sA);
    umma::copy_commit();
    uint32_t phase = 0, buf = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x, buf ^= 1) {
        // the next tile, into the buffer whose MMAs ended before the last epilogue
        if (item + (int)gridDim.x < nitems) load(item + gridDim.x, sA + (buf ^ 1) * TA);
        umma::copy_commit();
        umma::copy_wait<1>();
        umma::fence_async_smem();
        umma::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            umma::fence_after_sync();
            const uint32_t a0 = sA + buf * TA;
#pragma unroll
            for (int s = 0; s < K / 16; ++s)
                umma::mma_bf16(tmem, umma::smem_desc(a0 + 256 * s, 128, K * 16),
                               umma::smem_desc(sB + 256 * s, 128, K * 16), idesc, s > 0);
            umma::mma_commit(&mbar);
        }
        ok = __syncthreads_and(umma::mbar_wait(&mbar, phase, g.polls));
        if (!ok) break;
        phase ^= 1;
        umma::fence_after_sync();
        // ---- epilogue: warp w owns accumulator rows (TMEM lanes) 32w .. 32w+31 ----
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
        const int row0 = item * 128 + warp * 32;
        float inv = 0.f;
        if (g.off && row0 + lane < g.rows) inv = inv_degree(g.off[row0 + lane + 1] - g.off[row0 + lane]);
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            umma::tmem_ld16(trow + c0, v);
            store_rows(g, stage, row0, c0, inv, v);
        }
        umma::fence_before_sync();
        __syncthreads();  // the accumulator is read before the next tile's first MMA overwrites it
    }
    gemm_end(g, ok, &mbar, phase, tmem, NCOL);
}

// dW [m_valid x N] += A^T [m x vertices] times G [vertices x N]: an item is `chunk` vertices, 64 per step.
constexpr int kWgtK = 64, kWgtM = 128;
template <int N>
constexpr size_t wgt_smem() {
    return 2 * (size_t)(kWgtM + N) * kWgtK * 2;
}

template <int N>
__global__ void __launch_bounds__(kGemmThreads) k_gemm_wgt(GemmArgs g) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tslot;
    constexpr uint32_t TA = kWgtM * kWgtK * 2, TB = N * kWgtK * 2, NCOL = N < 32 ? 32 : N;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t tmem = gemm_begin(&mbar, &tslot, NCOL);
    constexpr uint32_t idesc = umma::idesc_bf16_f32(kWgtM, N) | umma::kMajorMN;
    const uint32_t sA = umma::smem_addr(smem), sB = sA + 2 * TA;
    const int nitems = (g.rows + g.chunk - 1) / g.chunk, MB = g.m_valid / 8;
    for (uint32_t i = tid; i < 2 * TA / 16; i += kGemmThreads)  // columns from m_valid on stay zero
        reinterpret_cast<uint4 *>(smem)[i] = zero4();
    __syncthreads();
    uint32_t phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        const int r0 = item * g.chunk, n = min(g.chunk, g.rows - r0), steps = (n + kWgtK - 1) / kWgtK;
        // vertex 8 kg + k of a step, 16-byte chunk c of its row: byte ((kg * chunks + c) * 8 + k) * 16
        auto load = [&](int step, uint32_t buf) {
            const int v0 = step * kWgtK;
            for (int q = tid; q < kWgtK * MB; q += kGemmThreads) {
                const int k = q & 7, c = (q >> 3) % MB, kg = (q >> 3) / MB, v = v0 + kg * 8 + k;
                umma::copy16(sA + buf * TA + ((kg * (kWgtM / 8) + c) * 8 + k) * 16,
                             g.A + (size_t)(r0 + min(v, n - 1)) * g.lda + c * 8, v < n);
            }
            for (int q = tid; q < kWgtK * (N / 8); q += kGemmThreads) {
                const int k = q & 7, c = (q >> 3) % (N / 8), v = v0 + (q >> 3) / (N / 8) * 8 + k;
                umma::copy16(sB + buf * TB + q * 16, g.B + (size_t)(r0 + min(v, n - 1)) * g.ldb + c * 8, v < n);
            }
        };
        load(0, 0);
        umma::copy_commit();
        for (int i = 0; i < steps; ++i) {
            if (i > 0) {  // the other buffer's MMAs
                ok = __syncthreads_and(umma::mbar_wait(&mbar, phase, g.polls));
                if (!ok) break;
                phase ^= 1;
            }
            if (i + 1 < steps) load(i + 1, (i + 1) & 1);
            umma::copy_commit();
            umma::copy_wait<1>();
            umma::fence_async_smem();
            umma::fence_before_sync();
            __syncthreads();
            if (tid == 0) {
                umma::fence_after_sync();
                const uint32_t a0 = sA + (i & 1) * TA, b0 = sB + (i & 1) * TB;
#pragma unroll
                for (int s = 0; s < kWgtK / 16; ++s)
                    umma::mma_bf16(tmem, umma::smem_desc(a0 + s * 2 * kWgtM * 16, kWgtM * 16, 128),
                                   umma::smem_desc(b0 + s * 2 * N * 16, N * 16, 128), idesc, i > 0 || s > 0);
                umma::mma_commit(&mbar);
            }
        }
        if (!ok) break;
        ok = __syncthreads_and(umma::mbar_wait(&mbar, phase, g.polls));
        if (!ok) break;
        phase ^= 1;
        umma::fence_after_sync();
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
        const int r = warp * 32 + lane;
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            umma::tmem_ld16(trow + c0, v);
            if (r < g.m_valid)
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (c0 + i < g.nb && v[i] != 0.0f) atomicAdd(&g.out_w[(size_t)r * g.nb + c0 + i], v[i]);
        }
        umma::fence_before_sync();
        __syncthreads();  // the accumulator is read before the next item's first MMA overwrites it
    }
    gemm_end(g, ok, &mbar, phase, tmem, NCOL);
}

// ------------------------------------------------------------------------------------ aggregation
// Sums over a vertex's neighbours, in row order (float32), of the first W 16-byte words of their row of
// `data` (row stride ld words).  Bound by L2: W * 16 bytes per arc.  Rows of at most kLongRow arcs: a group of
// lanes per vertex, eight rows in flight.  Longer rows: a block each; all threads stage tiles of kLongTile
// neighbours in shared memory while one thread per channel adds the previous tile (a chain of additions).  A
// hub of 70,000 arcs, walked by one warp with one row in flight, took 7.8 ms per pass; now 0.95 ms.  Mixed
// meshes and preferential attachment (27 M arcs, W = 8): 1.0 -> 0.78 ms, 4.5 TB/s of gathered rows.
constexpr int kLongTile = 128;

// A row walked by the block: add(tile, n) is called with each staged tile of n neighbours, in row order.
template <int W, typename Add>
__device__ __forceinline__ void long_row(const int32_t *__restrict__ col, int64_t b, int64_t e, const uint4 *data,
                                         int ld, uint4 (*tile)[kLongTile * W], Add add) {
    constexpr int kPer = (kLongTile * W + 255) / 256;  // words per thread and tile (256 threads)
    uint4 x[kPer];
    auto load = [&](int64_t j0) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int q = i * 256 + (int)threadIdx.x;
            const int64_t j = j0 + q / W;
            x[i] = zero4();
            if (q < kLongTile * W && j < e) x[i] = data[(size_t)__ldg(col + j) * ld + q % W];
        }
    };
    load(b);
    int par = 0;
    for (int64_t j0 = b; j0 < e; j0 += kLongTile, par ^= 1) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int q = i * 256 + (int)threadIdx.x;
            if (q < kLongTile * W) tile[par][q] = x[i];
        }
        __syncthreads();  // the tile is full; the other one's sum ended before this
        load(j0 + kLongTile);
        const int n = e - j0 < kLongTile ? (int)(e - j0) : kLongTile;
        add(reinterpret_cast<const char *>(tile[par]), n);
    }
}

// Right half of buf (row stride 2C) = bf16(mean over neighbours of the left half).
template <int C>
__global__ void __launch_bounds__(256) k_agg_fwd(const int64_t *__restrict__ off, const int32_t *__restrict__ col,
                                                 int nv, const int32_t *__restrict__ longrow, int nlong,
                                                 __nv_bfloat16 *buf) {
    constexpr int W = C / 8;  // 16-byte words of a row's left half
    __shared__ uint4 tile[2][kLongTile * W];
    if ((int)blockIdx.x < nlong) {
        const int v = longrow[blockIdx.x];
        const int64_t b = off[v], e = off[v + 1];
        float s = 0.f;
        long_row<W>(col, b, e, reinterpret_cast<const uint4 *>(buf), 2 * W, tile, [&](const char *t, int n) {
            if (threadIdx.x >= C) return;
            const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16 *>(t) + threadIdx.x;
            int i = 0;
            for (; i + 16 <= n; i += 16) {
                float y[16];
#pragma unroll
                for (int q = 0; q < 16; ++q) y[q] = __bfloat162float(x[(i + q) * C]);
#pragma unroll
                for (int q = 0; q < 16; ++q) s = __fadd_rn(s, y[q]);
            }
            for (; i < n; ++i) s = __fadd_rn(s, __bfloat162float(x[i * C]));
        });
        if (threadIdx.x < C)
            buf[(size_t)v * 2 * C + C + threadIdx.x] = __float2bfloat16_rn(__fmul_rn(s, inv_degree(e - b)));
        return;
    }
    constexpr int G = C / 2;   // lanes per vertex, two channels each
    constexpr int PW = 32 / G;  // vertices per warp
    const int lane = threadIdx.x & 31, sub = lane / G, sl = lane % G;
    const unsigned int *const words = reinterpret_cast<const unsigned int *>(buf);  // two channels each
    const int64_t gw = ((int64_t)(blockIdx.x - nlong) * blockDim.x + threadIdx.x) >> 5;
    const int64_t stride = ((int64_t)(gridDim.x - nlong) * blockDim.x >> 5) * PW;
    for (int64_t v0 = gw * PW; v0 < nv; v0 += stride) {
        const int64_t v = v0 + sub < nv ? v0 + sub : nv - 1;
        const int64_t s = off[v];
        const int deg = (int)(off[v + 1] - s);
        const bool mine = v0 + sub < nv && deg <= batch::kLongRow;
        const int len = mine ? deg : 0;
        int most = len;
        for (int o = G; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(DMOLP_FULL_MASK, most, o));
        float a0 = 0.f, a1 = 0.f;
        constexpr int U = G < 8 ? G : 8;
        for (int j0 = 0; j0 < most; j0 += G) {
            const int u = j0 + sl < len ? __ldg(col + s + j0 + sl) : -1;
            for (int j = 0; j < G && j0 + j < most; j += U) {
                unsigned int x[U];
                bool on[U];
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    const int uq = __shfl_sync(DMOLP_FULL_MASK, u, j + q, G);
                    on[q] = uq >= 0;
                    x[q] = on[q] ? words[(size_t)uq * C + sl] : 0u;
                }
#pragma unroll
                for (int q = 0; q < U; ++q)
                    if (on[q]) {
                        a0 = __fadd_rn(a0, __uint_as_float(x[q] << 16));
                        a1 = __fadd_rn(a1, __uint_as_float(x[q] & 0xffff0000u));
                    }
            }
        }
        if (mine) {
            const float inv = inv_degree(deg);
            *reinterpret_cast<__nv_bfloat162 *>(buf + (size_t)v * 2 * C + C + 2 * sl) =
                __floats2bfloat162_rn(__fmul_rn(a0, inv), __fmul_rn(a1, inv));
        }
    }
}

// Backward of one layer's input (64 channels): dH = dC[:, :64] + sum over neighbours v of dC[v, 64:] / deg(v)
// (the transpose of the mean for a symmetric graph; the data-gradient GEMM has divided its right half by the
// row's degree); G = bf16(dH * [H > 0]); db += column sums of G, one atomic per block and column.
__global__ void __launch_bounds__(256) k_agg_bwd(const int64_t *__restrict__ off, const int32_t *__restrict__ col,
                                                 int nv, const int32_t *__restrict__ longrow, int nlong,
                                                 const float *__restrict__ dC, const __nv_bfloat16 *__restrict__ H,
                                                 int ldh, __nv_bfloat16 *__restrict__ G, float *__restrict__ db) {
    extern __shared__ uint4 dyn[];
    __shared__ float cols[8][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto finish = [&](int64_t u, int c, float a, float h) {  // one channel
        const float g = h > 0.f ? __fadd_rn(dC[(size_t)u * 128 + c], a) : 0.f;
        return __float2bfloat16_rn(g);
    };
    if ((int)blockIdx.x < nlong) {
        const int u = longrow[blockIdx.x];
        const int64_t b = off[u], e = off[u + 1];
        float s = 0.f;
        long_row<16>(col, b, e, reinterpret_cast<const uint4 *>(dC) + 16, 32,
                     reinterpret_cast<uint4(*)[kLongTile * 16]>(dyn), [&](const char *t, int n) {
                         if (threadIdx.x >= 64) return;
                         const float *x = reinterpret_cast<const float *>(t) + threadIdx.x;
                         int i = 0;
                         for (; i + 16 <= n; i += 16) {
                             float y[16];
#pragma unroll
                             for (int q = 0; q < 16; ++q) y[q] = x[(i + q) * 64];
#pragma unroll
                             for (int q = 0; q < 16; ++q) s = __fadd_rn(s, y[q]);
                         }
                         for (; i < n; ++i) s = __fadd_rn(s, x[i * 64]);
                     });
        if (threadIdx.x < 64) {
            const int c = threadIdx.x;
            const __nv_bfloat16 q = finish(u, c, s, __bfloat162float(H[(size_t)u * ldh + c]));
            G[(size_t)u * 64 + c] = q;
            const float x = __bfloat162float(q);
            if (x != 0.f) atomicAdd(&db[c], x);
        }
        return;
    }
    const int64_t gw = ((int64_t)(blockIdx.x - nlong) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = (int64_t)(gridDim.x - nlong) * blockDim.x >> 5;
    const float2 *const pairs = reinterpret_cast<const float2 *>(dC);
    float s0 = 0.f, s1 = 0.f;
    for (int64_t u = gw; u < nv; u += nw) {
        const int64_t s = off[u];
        const int64_t deg = off[u + 1] - s;
        if (deg > batch::kLongRow) continue;
        const int len = (int)deg;
        float a0 = 0.f, a1 = 0.f;
        for (int j0 = 0; j0 < len; j0 += 32) {
            const int v = j0 + lane < len ? __ldg(col + s + j0 + lane) : -1;
            for (int j = 0; j < 32 && j0 + j < len; j += 8) {
                float2 x[8];
                bool on[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int vq = __shfl_sync(DMOLP_FULL_MASK, v, j + q);
                    on[q] = vq >= 0;
                    x[q] = on[q] ? pairs[(size_t)vq * 64 + 32 + lane] : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (on[q]) {
                        a0 = __fadd_rn(a0, x[q].x);
                        a1 = __fadd_rn(a1, x[q].y);
                    }
            }
        }
        const float2 l = pairs[(size_t)u * 64 + lane];
        const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(H + (size_t)u * ldh + 2 * lane);
        const float g0 = __bfloat162float(h.x) > 0.f ? __fadd_rn(l.x, a0) : 0.f;
        const float g1 = __bfloat162float(h.y) > 0.f ? __fadd_rn(l.y, a1) : 0.f;
        const __nv_bfloat162 q = __floats2bfloat162_rn(g0, g1);
        *reinterpret_cast<__nv_bfloat162 *>(G + (size_t)u * 64 + 2 * lane) = q;
        s0 += __bfloat162float(q.x);
        s1 += __bfloat162float(q.y);
    }
    cols[warp][2 * lane] = s0;
    cols[warp][2 * lane + 1] = s1;
    __syncthreads();
    if (threadIdx.x < 64) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += cols[w][threadIdx.x];
        if (t != 0.f) atomicAdd(&db[threadIdx.x], t);
    }
}

// Edge-contrastive loss over arcs (v, u): y * d2 + (1 - y) * max(0, margin - d2), y = same target label,
// d2 = |z_v - z_u|^2.  Four lanes per vertex (4 channels each).  G3 = bf16(dL/dz), db3 += its column sums.
__global__ void k_loss(const int64_t *__restrict__ off, const int32_t *__restrict__ col, int nv,
                       const float *__restrict__ Z, const int32_t *__restrict__ target, float scale,
                       __nv_bfloat16 *__restrict__ G, float *__restrict__ db, double *__restrict__ loss_sum) {
    const int lane = threadIdx.x & 31, sub = lane >> 2, q = lane & 3;
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t stride = ((int64_t)gridDim.x * blockDim.x >> 5) * 8;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    double ls = 0.0;
    for (int64_t v0 = gw * 8; v0 < nv; v0 += stride) {
        const int64_t v = v0 + sub;
        const bool act = v < nv;
        const int64_t b = act ? off[v] : 0, e = act ? off[v + 1] : 0;
        const float4 zv = act ? *reinterpret_cast<const float4 *>(Z + (size_t)v * 16 + 4 * q) : make_float4(0, 0, 0, 0);
        const int tv = act ? target[v] : 0;
        float g[4] = {0.f, 0.f, 0.f, 0.f};
        // every lane of the warp runs the longest row of its 8 vertices (the shuffles need all lanes)
        int64_t len = e - b, mx = len;
        for (int o = 4; o < 32; o <<= 1) mx = max(mx, (int64_t)__shfl_xor_sync(DMOLP_FULL_MASK, (long long)mx, o));
        for (int64_t t = 0; t < mx; ++t) {
            const bool on = t < len;
            const int u = on ? __ldg(col + b + t) : 0;
            float4 zu = make_float4(0, 0, 0, 0);
            if (on) zu = *reinterpret_cast<const float4 *>(Z + (size_t)u * 16 + 4 * q);
            const float d[4] = {__fsub_rn(zv.x, zu.x), __fsub_rn(zv.y, zu.y), __fsub_rn(zv.z, zu.z),
                                __fsub_rn(zv.w, zu.w)};
            float p = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) p = __fadd_rn(p, __fmul_rn(d[i], d[i]));
            p += __shfl_xor_sync(DMOLP_FULL_MASK, p, 1);
            p += __shfl_xor_sync(DMOLP_FULL_MASK, p, 2);
            if (on) {
                const bool y = target[u] == tv;
                const float coef = y ? 2.f : (p < kMargin ? -2.f : 0.f);
#pragma unroll
                for (int i = 0; i < 4; ++i) g[i] = __fadd_rn(g[i], __fmul_rn(coef, d[i]));
                if (q == 0) ls += y ? (double)p : (double)fmaxf(0.f, kMargin - p);
            }
        }
        if (act) {
            __align__(8) __nv_bfloat16 h[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                h[i] = __float2bfloat16_rn(__fmul_rn(g[i], scale));
                s[i] += __bfloat162float(h[i]);
            }
            *reinterpret_cast<uint2 *>(G + (size_t)v * 16 + 4 * q) = *reinterpret_cast<const uint2 *>(h);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (s[i] != 0.f) atomicAdd(&db[4 * q + i], s[i]);
    if (q == 0 && ls != 0.0) atomicAdd(loss_sum, ls);
}

// An upstream gradient given in FP32: G = bf16(dZ) [nv x 16], db += its column sums.
__global__ void k_grad_out(const float *dZ, int nv, __nv_bfloat16 *G, float *db) {
    const int c = threadIdx.x & 15;
    float s = 0.f;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)nv * 16;
         i += (int64_t)gridDim.x * blockDim.x) {
        const __nv_bfloat16 h = __float2bfloat16_rn(dZ[i]);
        G[i] = h;
        s += __bfloat162float(h);
    }
    if (s != 0.f) atomicAdd(&db[c], s);
}

__global__ void k_adam(float *p, const float *g, float *m, float *v, int n, float lr, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
}

__global__ void k_cast(const float *params, __nv_bfloat16 *W0, __nv_bfloat16 *W1, __nv_bfloat16 *W2,
                       __nv_bfloat16 *T0, __nv_bfloat16 *T1, __nv_bfloat16 *T2) {
    int o = 0;
    __nv_bfloat16 *W[3] = {W0, W1, W2}, *T[3] = {T0, T1, T2};
    const int Ks[3] = {2 * kIn, 2 * kHidden, 2 * kHidden}, Ns[3] = {kHidden, kHidden, kOut};
    for (int l = 0; l < 3; ++l) {
        const int K = Ks[l], N = Ns[l];
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K * N; i += gridDim.x * blockDim.x) {
            const int r = i / N, c = i % N;
            const __nv_bfloat16 h = __float2bfloat16_rn(params[o + i]);
            W[l][i] = h;
            T[l][c * K + r] = h;
        }
        o += K * N + N;
    }
}

// Gate scores: per graph, the mean of the network's output column 8 over its vertices (double sums).
__global__ void k_gate_scores(const float *Z, const int32_t *vinst, int nv, double *score) {
    const int lane = threadIdx.x & 31;
    for (int v0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); v0 < nv; v0 += gridDim.x * blockDim.x) {
        const int v = v0 + lane;
        const int i = v < nv ? vinst[v] : -1;
        double x = v < nv ? (double)Z[(size_t)v * 16 + 8] : 0.0;
        const int i0 = __shfl_sync(DMOLP_FULL_MASK, i, 0);
        if (__all_sync(DMOLP_FULL_MASK, i == i0)) {
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(DMOLP_FULL_MASK, x, o);
            if (lane == 0) atomicAdd(&score[i0], x);
        } else if (i >= 0) {
            atomicAdd(&score[i], x);
        }
    }
}

// Upstream gradient of the gate loss: column 8 of vertex v gets g[graph of v], the other columns 0.
__global__ void k_gate_grad(const float *g, const int32_t *vinst, int nv, float *dZ) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)nv * 16;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = i >> 4;
        dZ[i] = (i & 15) == 8 ? g[vinst[v]] : 0.f;
    }
}

// Proposal coordinates: random-walk features + the network's first 8 outputs (its residual); 16 wide, the
// upper 8 columns 0.
__global__ void k_coords(const float *__restrict__ Xf, const float *__restrict__ Z, int nv, float *__restrict__ P) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)nv * 16;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = i >> 4;
        const int j = (int)(i & 15);
        P[i] = j < 8 ? __fadd_rn(Xf[v * 16 + 2 + j], Z[v * 16 + j]) : 0.f;
    }
}

template <int N, int K>
void launch_rows(const GemmArgs &g, int num_sms, cudaStream_t s) {
    using R = RowGemm<N, K>;
    cudaFuncSetAttribute(k_gemm_rows<N, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)R::kSmem);
    const int grid = std::max(1, std::min((g.rows + 127) / 128, num_sms * R::kPerSm));
    k_gemm_rows<N, K><<<grid, kGemmThreads, R::kSmem, s>>>(g);
}

template <int N>
void launch_wgt(const GemmArgs &g, int num_sms, cudaStream_t s) {
    cudaFuncSetAttribute(k_gemm_wgt<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wgt_smem<N>());
    const int grid = std::max(1, std::min((g.rows + g.chunk - 1) / g.chunk, num_sms * 4));
    k_gemm_wgt<N><<<grid, kGemmThreads, wgt_smem<N>(), s>>>(g);
}

inline int grid_for(int64_t n, int num_sms) {
    const int64_t b = (n + 255) / 256;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)num_sms * 16));
}

}  // namespace

void gemm(const GemmArgs &g, int n, int num_sms, cudaStream_t s) {
    if (g.rows <= 0) return;
    if (g.kind == kBwdWeight) {
        if (n == 64) launch_wgt<64>(g, num_sms, s);
        else launch_wgt<16>(g, num_sms, s);
    } else if (n == 64) {
        if (g.K == 32) launch_rows<64, 32>(g, num_sms, s);
        else launch_rows<64, 128>(g, num_sms, s);
    } else if (n == 16) {
        launch_rows<16, 128>(g, num_sms, s);
    } else {
        if (g.K == 16) launch_rows<128, 16>(g, num_sms, s);
        else launch_rows<128, 64>(g, num_sms, s);
    }
}

void agg_fwd(const batch::View &b, __nv_bfloat16 *buf, int C) {
    const int nv = (int)b.nv;
    const int grid = b.nlong + grid_for((int64_t)nv * (C / 2), b.num_sms);
    if (C == 16) k_agg_fwd<16><<<grid, 256, 0, b.stream>>>(b.off, b.col, nv, b.longrow, b.nlong, buf);
    else k_agg_fwd<64><<<grid, 256, 0, b.stream>>>(b.off, b.col, nv, b.longrow, b.nlong, buf);
}

void agg_bwd(const batch::View &b, const float *dC, const __nv_bfloat16 *Hbuf, int ldh, __nv_bfloat16 *G, float *db) {
    const int nv = (int)b.nv;
    // The limit is the kernel's, not the launch's: the same value in every call, or a thread whose batch has no long
    // rows could lower it between another's setting and its launch.
    constexpr size_t kTiles = 2 * kLongTile * 16 * sizeof(uint4);
    cudaFuncSetAttribute(k_agg_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTiles);
    const size_t smem = b.nlong > 0 ? kTiles : 0;
    k_agg_bwd<<<b.nlong + grid_for((int64_t)nv * 32, b.num_sms), 256, smem, b.stream>>>(b.off, b.col, nv, b.longrow,
                                                                                       b.nlong, dC, Hbuf, ldh, G, db);
}

void loss(const int64_t *off, const int32_t *col, int nv, const float *Z, const int32_t *target, double inv_arcs,
          __nv_bfloat16 *G, float *db, double *loss_sum, int num_sms, cudaStream_t s) {
    k_loss<<<grid_for((int64_t)nv * 4, num_sms), 256, 0, s>>>(off, col, nv, Z, target, (float)(2.0 * inv_arcs), G,
                                                             db, loss_sum);
}

void grad_out(const float *dZ, int nv, __nv_bfloat16 *G, float *db, int num_sms, cudaStream_t s) {
    k_grad_out<<<grid_for((int64_t)nv * 16, num_sms), 256, 0, s>>>(dZ, nv, G, db);
}

void adam(float *p, const float *g, float *m, float *v, int n, float lr, int step, cudaStream_t s) {
    const float c1 = 1.f - powf(0.9f, (float)step), c2 = 1.f - powf(0.999f, (float)step);
    k_adam<<<(n + 255) / 256, 256, 0, s>>>(p, g, m, v, n, lr, c1, c2);
}

void cast_weights(const float *params, __nv_bfloat16 *const W[3], __nv_bfloat16 *const Wt[3], cudaStream_t s) {
    k_cast<<<32, 256, 0, s>>>(params, W[0], W[1], W[2], Wt[0], Wt[1], Wt[2]);
}

void gate_scores(const float *Z, const int32_t *vinst, int nv, double *score, int num_sms, cudaStream_t s) {
    k_gate_scores<<<grid_for(nv, num_sms), 256, 0, s>>>(Z, vinst, nv, score);
}

void gate_grad(const float *g, const int32_t *vinst, int nv, float *dZ, int num_sms, cudaStream_t s) {
    k_gate_grad<<<grid_for((int64_t)nv * 16, num_sms), 256, 0, s>>>(g, vinst, nv, dZ);
}

void coords(const float *Xf, const float *Z, int nv, float *P, int num_sms, cudaStream_t s) {
    k_coords<<<grid_for((int64_t)nv * 16, num_sms), 256, 0, s>>>(Xf, Z, nv, P);
}

}  // namespace mpnn
}  // namespace dmolp
