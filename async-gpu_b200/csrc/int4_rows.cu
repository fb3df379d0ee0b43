// Group-wise int4 weight-only Linear of three to eight f32 rows in one kernel (the stand-alone Linear; a model's chain of
// kernels keeps fp16 activations and the tcgen05 GEMM, which starts under its predecessor: GPT-2 XL steps of eight
// sequences 1.26 ms that way, 2.2 ms with this kernel, whose blocks fill the SMs' registers).
//
// So few rows leave the tcgen05 GEMM (gemm_tc.cu) waiting on its own start, and on a launch of its own that converts the
// rows.  Here a warp multiplies 16 features by mma.sync straight from registers: two 16-byte loads per lane are 16 features
// x 128 inputs, requested before the wait on the previous kernel (weights do not depend on it), unpacked to exact fp16
// integers, multiplied with the rows as the MMA's eight columns, and scaled in f32 once per 128 inputs.  Every block rounds
// its part of the rows to fp16 while it stages them in shared memory, a warp per row.
//
// K is dealt out to the warps that share a tile and to the blocks of a cluster, which store their sums into the first one's
// shared memory (fixed order).  Bound: latencies (one load, a few MMAs, the reduction); mma.sync has an eighth of
// tcgen05's rate on this GPU, so wide outputs and more rows stay with the GEMM.  Eight rows, back to back, conversion + GEMM / this
// kernel: 768 x 3072 5.9 / 3.6 us, 3072 x 768 6.1 / 4.2, 1600 x 4800 6.4 / 5.5; 768 x 50257 12.8 / 12.9 (not taken).
//
// y[m,n] = sum_k fp16(x[m,k]) * (nibble(k,n)-8) * scale[k/group,n] (+ bias[n]): int4_linear.rs:72-134.
#include <algorithm>

#include "device_utils.cuh"

namespace {

constexpr int THREADS = 256, WARPS = THREADS / 32, AHEAD = 3, ROWS = 8, MAX_TPB = 4;

__device__ __forceinline__ void mma_f16(float (&d)[4], __half2 a0, __half2 a1, __half2 a2, __half2 a3, uint32_t b0, uint32_t b1) {
    auto u = [](__half2 h) { return *reinterpret_cast<uint32_t *>(&h); };
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(u(a0)), "r"(u(a1)), "r"(u(a2)), "r"(u(a3)), "r"(b0), "r"(b1));
}
// Where eight inputs k .. k+7 (k a multiple of 8) of a staged row lie: within 128, word i of plane t after word i of the
// planes before it, so that the four lanes of a row read 64 neighbouring bytes.
__device__ __forceinline__ int staged_at(int k) { return (k & ~127) + ((k >> 3) & 3) * 32 + ((k >> 5) & 3) * 8; }
__device__ __forceinline__ uint4 halves8(float4 a, float4 b) {
    return make_uint4(pack_f16x2(a.x, a.y), pack_f16x2(a.z, a.w), pack_f16x2(b.x, b.y), pack_f16x2(b.z, b.w));
}

// grid (groups of TPB tiles of 16 features, splits), cluster (1, splits, 1); KS warps share a tile's part of K.
template <int TPB>
__global__ void __launch_bounds__(THREADS, 2)
int4_rows_kernel(const uint8_t *__restrict__ tiles, const __half *__restrict__ scales, Fresh<float> x, int M, int K, int N, int k_blocks,
                 int n_pad, int group_units, int units_per_split, Epilogue epi) {
    constexpr int KS = WARPS / TPB, SUMS = TPB * 16 * ROWS; // warps of a tile, sums of the block
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
    const int split = blockIdx.y, splits = gridDim.y;
    const int u0 = split * units_per_split, units = min(units_per_split, (k_blocks + 1) / 2 - u0); // of 128 inputs
    const int ldx = units_per_split * 128 + 32; // halves; rows 64 bytes apart modulo 128
    __half *xs = reinterpret_cast<__half *>(smem);
    float *red = reinterpret_cast<float *>(xs + ROWS * ldx);  // [KS][TPB][ROWS][16]
    float *part = red + KS * SUMS;                            // [splits][SUMS] in the cluster's first block
    pdl_trigger();
    if (splits > 1) cluster_arrive(); // waited for before the first store into another block

    const int slice = warp % KS, tile_in = warp / KS, tile = blockIdx.x * TPB + tile_in;
    const uint8_t *src = tiles + (size_t)(tile >> 3) * k_blocks * TILE_BYTES + (tq & 1) * 2048 + ((tile & 7) * 16 + gq) * 16;
    uint4 wa[AHEAD], wb[AHEAD];
    float sa[AHEAD], sb[AHEAD];
    auto load = [&](int i, int u) { // unit u of the block's range
        const int kb = 2 * (u0 + u) + (tq >> 1);
        wa[i] = wb[i] = make_uint4(0x88888888u, 0x88888888u, 0x88888888u, 0x88888888u); // zeros
        sa[i] = sb[i] = 0.0f;
        if (u >= units || tile * 16 >= n_pad) return;
        if (kb < k_blocks) {
            const uint8_t *p = src + (size_t)kb * TILE_BYTES;
            wa[i] = __ldg(reinterpret_cast<const uint4 *>(p));
            wb[i] = __ldg(reinterpret_cast<const uint4 *>(p + 128));
        }
        const __half *s = scales + (size_t)((u0 + u) / group_units) * n_pad + tile * 16 + gq;
        sa[i] = __half2float(s[0]);
        sb[i] = __half2float(s[8]);
    };
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) load(i, slice + i * KS);

    // ---- the rows' part of K as fp16, zeros past it and past M ----
    const int k_from = u0 * 128, groups = units * 16; // of eight inputs
    {
        constexpr int U = 4; // groups of a lane in flight
        const Fresh<float> row = x + (size_t)(warp < M ? warp : 0) * K + k_from;
        __half *to = xs + warp * ldx;
        const int have = warp < M ? min(groups, (K - k_from) / 8) : 0;
        pdl_wait();
        for (int g0 = lane; g0 < groups; g0 += U * 32) {
            uint4 h[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int g = g0 + u * 32;
                h[u] = g < have ? halves8(row.four((size_t)g * 8), row.four((size_t)g * 8 + 4)) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (g0 + u * 32 < groups) *reinterpret_cast<uint4 *>(to + staged_at((g0 + u * 32) * 8)) = h[u];
        }
    }
    __syncthreads();

    // ---- products ----
    float tot[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int n0 = slice; n0 < units; n0 += AHEAD * KS) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int u = n0 + i * KS;
            if (u >= units) break; // warp-uniform
            const uint32_t qa[4] = {wa[i].x, wa[i].y, wa[i].z, wa[i].w}, qb[4] = {wb[i].x, wb[i].y, wb[i].z, wb[i].w};
            const float s0 = sa[i], s1 = sb[i];
            load(i, u + AHEAD * KS);
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                __half2 a[4], b[4];
                unpack8_int4(qa[w], a);
                unpack8_int4(qb[w], b);
                const uint4 xv = *reinterpret_cast<const uint4 *>(xs + gq * ldx + u * 128 + w * 32 + tq * 8);
                mma_f16(acc, a[0], b[0], a[1], b[1], xv.x, xv.y);
                mma_f16(acc, a[2], b[2], a[3], b[3], xv.z, xv.w);
            }
            tot[0] = fmaf(s0, acc[0], tot[0]);
            tot[1] = fmaf(s0, acc[1], tot[1]);
            tot[2] = fmaf(s1, acc[2], tot[2]);
            tot[3] = fmaf(s1, acc[3], tot[3]);
        }
    }
    { // features gq and gq + 8, rows 2 tq and 2 tq + 1
        float *r = red + ((size_t)(slice * TPB + tile_in) * ROWS + 2 * tq) * 16 + gq;
        r[0] = tot[0];
        r[16] = tot[1];
        r[8] = tot[2];
        r[24] = tot[3];
    }
    __syncthreads();

    // ---- sums of the slices, of the cluster, epilogue: thread v has row v / (16 TPB), feature v % (16 TPB) ----
    constexpr int PER = (SUMS + THREADS - 1) / THREADS;
    float sum[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int v = tid + j * THREADS, m = v / (16 * TPB), f = v % (16 * TPB);
        sum[j] = 0.0f;
        if (v < SUMS)
#pragma unroll
            for (int s = 0; s < KS; ++s) sum[j] += red[((size_t)(s * TPB + (f >> 4)) * ROWS + m) * 16 + (f & 15)];
    }
    if (splits > 1) {
        cluster_wait();
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (tid + j * THREADS < SUMS) st_cluster(&part[split * SUMS + tid + j * THREADS], 0, sum[j]);
        cluster_arrive();
        cluster_wait(); // every block's sums are in the first block
        if (split != 0) return;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int v = tid + j * THREADS;
            sum[j] = 0.0f;
            if (v < SUMS)
                for (int s = 0; s < splits; ++s) sum[j] += part[s * SUMS + v]; // fixed order
        }
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int v = tid + j * THREADS, m = v / (16 * TPB), n = blockIdx.x * 16 * TPB + v % (16 * TPB);
        if (v >= SUMS || m >= M) continue;
        if (n < N) epi_apply(epi, m, n, sum[j]);
    }
}

struct RowsPlan {
    int tpb, blocks, splits, per;
    size_t smem;
};
// Tiles per block: as few as leave two blocks per SM at most (a warp then has few units, all requested at the start).
// Then K is split over a cluster while there are places left, down to a unit per warp.
RowsPlan rows_plan(const b200nn_ctx *ctx, const Int4Weight &w) {
    RowsPlan p;
    const int tiles = (w.N + 15) / 16, units = (w.k_blocks + 1) / 2, slots = 2 * ctx->sm_count;
    p.tpb = 1;
    while (p.tpb < 2 * MAX_TPB && (tiles + p.tpb - 1) / p.tpb > slots) p.tpb *= 2;
    p.blocks = (tiles + p.tpb - 1) / p.tpb;
    const int ks = std::max(1, WARPS / p.tpb);
    p.splits = std::max(1, std::min({8, slots / p.blocks, units / ks}));
    p.per = (units + p.splits - 1) / p.splits;
    p.splits = (units + p.per - 1) / p.per;
    p.smem = (size_t)ROWS * (p.per * 128 + 32) * 2 + (size_t)(ks + (p.splits > 1 ? p.splits : 0)) * p.tpb * 16 * ROWS * 4;
    return p;
}

template <int TPB>
int rows_launch(b200nn_ctx *ctx, const Int4Weight &w, const float *x, int M, const RowsPlan &p, const Epilogue &epi) {
    auto kern = int4_rows_kernel<TPB>;
    static bool attr_done[16] = {}; // function attributes are per device
    if (!attr_done[ctx->device & 15]) {
        CK(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
        prefer_max_smem(kern);
        attr_done[ctx->device & 15] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.blocks, p.splits);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = p.splits;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = ctx->pdl ? attr : attr + 1;
    cfg.numAttrs = (ctx->pdl ? 1 : 0) + (p.splits > 1 ? 1 : 0);
    CK(ctx, cudaLaunchKernelEx(&cfg, kern, (const uint8_t *)w.tiled->p, (const __half *)w.scales_h->p, Fresh<float>(x), M, w.K, w.N, w.k_blocks,
                               w.n_pad, w.group / 128, p.per, epi));
    CK_LAUNCH(ctx, "int4_rows_kernel");
    return B200NN_OK;
}

}  // namespace

// Not for more tiles than four per block leave, nor for parts of K whose rows take longer to stage than the GEMM's start
// (6400 x 1600, eight rows: 8.1 us conversion + GEMM, 8.5 us here; four rows 7.9 and 7.3).  Blocks of several tiles fill the GPU
// without a split of K, and a warp's units then come one after another; weights beyond L2, conversion + GEMM / here, us.  Two
// tiles: 2048 x 6400 8 rows 7.9 / 7.1, 3072 x 6400 4 rows 9.2 / 9.4, 5 rows 8.9 / 9.6, 4096 x 6400 4 rows 10.1 / 12.3.  Four: 1280 x 9500
// 8 rows 7.5 / 7.2, 1600 x 9500 4 rows 8.4 / 8.5, 8 rows 8.3 / 9.0, 2048 x 9500 4 rows 9.2 / 10.1.
bool int4_rows_supported(const b200nn_ctx *ctx, const Int4Weight &w, const float *x, int M) {
    if (!w.fast || w.group % 128 != 0 || M <= std::max(2, ctx->gemv_max_rows) || M > ctx->int4_rows_max || ((uintptr_t)x & 15)) return false;
    const RowsPlan p = rows_plan(ctx, w);
    const int most = p.tpb == 1 ? 128 : p.tpb == 2 ? (M <= 4 ? 24 : 16) : M <= 4 ? 13 : 10; // units of 128 inputs per block
    return p.tpb <= MAX_TPB && M * p.per <= 128 && p.per <= most;
}

int launch_int4_rows(b200nn_ctx *ctx, const Int4Weight &w, const float *x, int M, const Epilogue &epi) {
    const RowsPlan p = rows_plan(ctx, w);
    return p.tpb == 1 ? rows_launch<1>(ctx, w, x, M, p, epi) : p.tpb == 2 ? rows_launch<2>(ctx, w, x, M, p, epi) : rows_launch<4>(ctx, w, x, M, p, epi);
}
