// f32 Linear (y = x * W + b with W stored [K,N]) on CUDA cores with the shared fused epilogue.
// Replaces the reference's matmul dispatch + bias_add pair (ops/gemm.rs:20-299, reshape.rs:112-156)
// for the f32 model family.  Two kernels:
//   f32_gemv_kernel  M <= 4 rows: weights read once, 32 columns per block, K split over the block's warps
//                    and the blocks of a cluster (fixed order of sums).
//   f32_gemm_kernel  64x64x16 shared-memory tiles, 4x4 outputs per thread, any M.
#include <algorithm>

#include "device_utils.cuh"

static constexpr int FGEMV_THREADS = 256;
static constexpr int FGEMV_AHEAD = 12;         // weight loads a thread has in flight
static constexpr size_t FGEMV_XS = 160 * 1024; // bytes of activations a block holds at a time

// grid (column tiles, splits), cluster (1, splits, 1).  A decode step of one sequence is bound by the weights'
// bytes and by the hand-over from kernel to kernel, so: the block's tile is narrow and its K range short enough that
// most of its weights are requested before the wait on the previous kernel (they are constants), 16 bytes per
// lane (VEC 4: eight lanes per row, 32 K slices in a block; VEC 1, rows that do not start on 16 bytes: eight slices).
// The partial sums of a cluster are stored into its first block's shared memory, one barrier, no scratch in memory.
// With `ln.g` the activations are the LayerNorm of the f32 rows x: every block takes the statistics of the whole
// row itself, which saves a kernel between two Linears (norm_rows_to_smem).
// PIECES: K ranges whose activations exceed x_rows rows (whole trips of the loop) are staged piece by piece.  One row,
// 100000 x 64: 11 ms on the tiled kernel, which has one block per 64 columns, 28 us here.
// COLS: 32 columns, one 128-byte line of every weight row, or 128 for a weight that would have more than three blocks per
// SM that way (an output matrix), each paying for its start and its activations (768 x 50257 with one / four rows: 65 / 147 us
// in 32 columns, 44 / 65 in 128; 100 x 50257: 21 / 40 and 14 / 15).  Those are never split over a cluster and take no LayerNorm.
// GPT-2 Small, one sequence, 64 tokens after a prompt of 64: 52.5 ms with 4-byte loads, four in flight, plain launches and
// a reduction through memory, 24.7 ms with this.
template <int MT, int VEC, int COLS, bool PIECES, typename XT>
__global__ void __launch_bounds__(FGEMV_THREADS)
f32_gemv_kernel(const float *__restrict__ w, int ldw, Fresh<XT> x, int m_valid, int m0, int K, int N, int k_per_split, int x_rows,
                NormIn ln, Epilogue epi) {
    constexpr int LANES = COLS / VEC;                   // lanes across a row of the tile
    constexpr int SLICES = FGEMV_THREADS / LANES, WARPS = FGEMV_THREADS / 32, TRIP = FGEMV_AHEAD * SLICES;
    extern __shared__ float smem_f[];
    const int split = blockIdx.y, splits = gridDim.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slice = tid / LANES, c = (tid % LANES) * VEC, n_base = blockIdx.x * COLS;
    const int k0 = split * k_per_split, rows = min(k_per_split, K - k0);
    float *xs = smem_f;                                 // [MT][x_rows] activations of this block's K range
    float *red = xs + MT * x_rows;                      // [WARPS][MT][COLS]
    float *part = red + WARPS * MT * COLS;              // [splits][MT][COLS] in the cluster's first block
    pdl_trigger();
    if (splits > 1) cluster_arrive(); // waited for before the first store into another block

    const float *wp = w + (size_t)(k0 + slice) * ldw + n_base + c;
    const bool n_ok = n_base + c < (VEC == 4 ? ldw : N);
    float buf[FGEMV_AHEAD][VEC];
    auto load = [&](float (&v)[VEC], int r) { // row `slice + r` of the range
        if (!n_ok || slice + r >= rows) return;
        if constexpr (VEC == 4) {
            const float4 t = __ldg(reinterpret_cast<const float4 *>(wp + (size_t)r * ldw));
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
            v[0] = __ldg(wp + (size_t)r * ldw);
        }
    };
#pragma unroll
    for (int j = 0; j < FGEMV_AHEAD; ++j) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) buf[j][i] = 0.0f;
        load(buf[j], j * SLICES);
    }
    if constexpr (sizeof(XT) == 4 && COLS == 32) {
        if (ln.g) norm_rows_to_smem<MT, FGEMV_THREADS>(ln, x, m_valid, K, k0, rows, x_rows, xs, red);
    }
    if (sizeof(XT) != 4 || COLS != 32 || !ln.g) {
        pdl_wait();
        rows_to_smem<MT, FGEMV_THREADS>(x, m_valid, K, k0, PIECES ? min(rows, x_rows) : rows, x_rows, xs);
    }
    __syncthreads();

    float acc[MT][VEC];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[m][i] = 0.0f;
    int piece = 0; // first row of the range in xs
    for (int r0 = 0; r0 < rows; r0 += TRIP) {
        if (PIECES && r0 == piece + x_rows) {
            piece = r0;
            __syncthreads();
            rows_to_smem<MT, FGEMV_THREADS>(x, m_valid, K, k0 + r0, min(rows - r0, x_rows), x_rows, xs);
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < FGEMV_AHEAD; ++j) {
            const int r = r0 + j * SLICES;
            if (slice + r < rows) {
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const float xv = xs[m * x_rows + slice + r - piece];
#pragma unroll
                    for (int i = 0; i < VEC; ++i) acc[m][i] = fmaf(xv, buf[j][i], acc[m][i]);
                }
            }
            load(buf[j], r + TRIP);
        }
    }
    // the four K slices of a warp by shuffles, the warps through shared memory, the blocks of the cluster in its first
    if constexpr (LANES == 8) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int i = 0; i < VEC; ++i) {
                acc[m][i] += __shfl_xor_sync(0xffffffffu, acc[m][i], 8);
                acc[m][i] += __shfl_xor_sync(0xffffffffu, acc[m][i], 16);
            }
    }
    if (lane < LANES)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int i = 0; i < VEC; ++i) red[(warp * MT + m) * COLS + c + i] = acc[m][i];
    __syncthreads();
    if constexpr (COLS > 32) {
        for (int o = tid; o < MT * COLS; o += FGEMV_THREADS) { // a warp: 32 consecutive features of a row
            const int m = o / COLS, n = n_base + o % COLS;
            if (m >= m_valid) break;
            float t = 0.0f;
#pragma unroll
            for (int s = 0; s < WARPS; ++s) t += red[s * MT * COLS + o];
            if (n < N) epi_apply(epi, m0 + m, n, t);
            if (epi.amax_val) epi_argmax1(epi, m0 + m, n, t + (epi.bias && n < N ? epi.bias[n] : 0.0f), n < N);
        }
        return;
    }
    float t = 0.0f;
    if (warp < MT)
#pragma unroll
        for (int s = 0; s < WARPS; ++s) t += red[(s * MT + warp) * COLS + lane];
    if (splits > 1) {
        cluster_wait();
        if (warp < MT) st_cluster(&part[(split * MT + warp) * COLS + lane], 0, t);
        cluster_arrive();
        cluster_wait(); // every block's sums are in the first block
        if (split != 0) return;
        t = 0.0f;
        if (warp < MT)
            for (int sp = 0; sp < splits; ++sp) t += part[(sp * MT + warp) * COLS + lane];
    }
    if (warp < min(MT, m_valid)) { // one warp per row: 32 consecutive features
        const int n = n_base + lane;
        if (n < N) epi_apply(epi, m0 + warp, n, t);
        if (epi.amax_val) epi_argmax1(epi, m0 + warp, n, t + (epi.bias && n < N ? epi.bias[n] : 0.0f), n < N);
    }
}

template <typename XT>
__global__ void __launch_bounds__(256)
f32_gemm_kernel(const float *__restrict__ w, int ldw, const XT *__restrict__ x, int M, int K, int N, Epilogue epi) {
    __shared__ float xs[16][64 + 1]; // [k][m]
    __shared__ float ws[16][64];     // [k][n]
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m_base = blockIdx.y * 64, n_base = blockIdx.x * 64;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        for (int i = threadIdx.x; i < 64 * 16; i += 256) {
            int mm = i >> 4, kk = i & 15; // consecutive threads walk k: contiguous in x
            int m = m_base + mm, k = k0 + kk;
            xs[kk][mm] = (m < M && k < K) ? load_as_float<XT>(x, (size_t)m * K + k) : 0.0f;
        }
        for (int i = threadIdx.x; i < 16 * 64; i += 256) {
            int kk = i >> 6, nn = i & 63;
            int k = k0 + kk, n = n_base + nn;
            ws[kk][nn] = (k < K && n < N) ? w[(size_t)k * ldw + n] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int m = m_base + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int n = n_base + tx + 16 * j;
            if (n < N) epi_apply(epi, m, n, acc[i][j]);
        }
    }
}

template <int MT, int VEC, int COLS, bool PIECES, typename XT>
static int f32_gemv_launch(b200nn_ctx *ctx, const F32Weight &w, const XT *x, int m_valid, int m0, int splits, int per, int x_rows, const NormIn &ln,
                           const Epilogue &epi) {
    const int tiles = (w.N + COLS - 1) / COLS;
    auto kern = f32_gemv_kernel<MT, VEC, COLS, PIECES, XT>;
    const size_t smem = ((size_t)MT * x_rows + (size_t)(FGEMV_THREADS / 32 + splits) * MT * COLS) * sizeof(float);
    static bool attr_done[16] = {}; // function attributes are per device
    if (!attr_done[ctx->device & 15]) {
        CK(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        prefer_max_smem(kern);
        attr_done[ctx->device & 15] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, splits);
    cfg.blockDim = dim3(FGEMV_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = splits;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl && !w.volatile_w ? 2 : 1;
    CK(ctx, cudaLaunchKernelEx(&cfg, kern, (const float *)w.w_kn->p, w.ld(), x, m_valid, m0, w.K, w.N, per, x_rows, ln, epi));
    CK_LAUNCH(ctx, "f32_gemv_kernel");
    return B200NN_OK;
}
template <int MT, int VEC, int COLS, typename XT>
static int f32_gemv_plan(b200nn_ctx *ctx, const F32Weight &w, const XT *x, int m_valid, int m0, const NormIn &ln, const Epilogue &epi) {
    // K split over a cluster until there is about a block per SM (GPT-2 Small, 64 tokens after a prompt of 64: 24.7 ms; two
    // blocks per SM 27.0, three 27.6), none of under 64 rows; activations of a longer range are staged in whole trips
    constexpr int TRIP = FGEMV_AHEAD * FGEMV_THREADS * VEC / COLS, X_ROWS = (int)(FGEMV_XS / (MT * sizeof(float))) / TRIP * TRIP;
    const int tiles = (w.N + COLS - 1) / COLS;
    int splits = COLS > 32 ? 1 : std::min(8, std::max(1, ctx->sm_count / tiles));
    splits = std::min(splits, std::max(1, w.K / 64));
    const int per = (w.K + splits - 1) / splits;
    splits = (w.K + per - 1) / per;
    if (per <= X_ROWS) return f32_gemv_launch<MT, VEC, COLS, false, XT>(ctx, w, x, m_valid, m0, splits, per, per, ln, epi);
    return f32_gemv_launch<MT, VEC, COLS, true, XT>(ctx, w, x, m_valid, m0, splits, per, X_ROWS, ln, epi);
}
template <int MT, typename XT>
static int f32_gemv_chunk(b200nn_ctx *ctx, const F32Weight &w, const XT *x, int m_valid, int m0, const NormIn &ln, const Epilogue &epi) {
    // rows of the weight that all start on 16 bytes: vector loads
    if (w.ld() % 4 == 0 && !((uintptr_t)w.w_kn->p & 15))
        return !ln.g && w.N > 3 * 32 * ctx->sm_count ? f32_gemv_plan<MT, 4, 128, XT>(ctx, w, x, m_valid, m0, ln, epi)
                                                     : f32_gemv_plan<MT, 4, 32, XT>(ctx, w, x, m_valid, m0, ln, epi);
    return f32_gemv_plan<MT, 1, 32, XT>(ctx, w, x, m_valid, m0, ln, epi);
}

template <typename XT>
static int f32_linear_t(b200nn_ctx *ctx, const F32Weight &w, const XT *x, int M, const NormIn &ln, const Epilogue &epi) {
    if (M <= F32_GEMV_ROWS) {
        if (M == 4) return f32_gemv_chunk<4, XT>(ctx, w, x, 4, 0, ln, epi);
        if (M >= 2) {
            TRY((f32_gemv_chunk<2, XT>(ctx, w, x, 2, 0, ln, epi)));
            if (M == 3) return f32_gemv_chunk<1, XT>(ctx, w, x + (size_t)2 * w.K, 1, 2, ln, epi);
            return B200NN_OK;
        }
        return f32_gemv_chunk<1, XT>(ctx, w, x, 1, 0, ln, epi);
    }
    dim3 grid((w.N + 63) / 64, (M + 63) / 64);
    PREFER_SMEM_ONCE(f32_gemm_kernel<XT>);
    f32_gemm_kernel<XT><<<grid, 256, 0, ctx->stream>>>((const float *)w.w_kn->p, w.ld(), x, M, w.K, w.N, epi);
    CK_LAUNCH(ctx, "f32_gemm_kernel");
    return B200NN_OK;
}

bool f32_linear_takes_norm(const F32Weight &w, int M) { return M >= 1 && M <= F32_GEMV_ROWS && w.K <= NORM_IN_MAX; }

int launch_f32_linear(b200nn_ctx *ctx, const F32Weight &w, const void *x, bool x_half, int M, const Epilogue &epi, const NormIn &ln) {
    if (M <= 0) return B200NN_OK;
    if (ln.g) {
        if (x_half || !f32_linear_takes_norm(w, M))
            return set_error(ctx, B200NN_ERR_UNSUPPORTED, "f32 Linear: only the GEMV of few rows takes a LayerNorm with its input");
        return f32_linear_t<float>(ctx, w, (const float *)x, M, ln, epi);
    }
    if (f16_gemm_tc_supported(ctx, w, M) && !((uintptr_t)x & 15)) {
        // more than four rows: fp16 operands on the tensor cores.  f32 activations are converted once
        // into a buffer the context keeps (grown outside stream capture only).
        if (x_half) return launch_f16_gemm_tc(ctx, w, (const __half *)x, M, epi);
        const size_t need = (size_t)M * w.K * sizeof(__half);
        if (!ctx->xh || ctx->xh->bytes < need) {
            if (ctx->capturing) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "activation buffer cannot grow during graph capture");
            ctx->xh.reset();
            TRY(dev_alloc(ctx, need, &ctx->xh));
        }
        TRY(launch_f32_to_half(ctx, (const float *)x, (__half *)ctx->xh->p, (size_t)M * w.K));
        return launch_f16_gemm_tc(ctx, w, (const __half *)ctx->xh->p, M, epi);
    }
    return x_half ? f32_linear_t<__half>(ctx, w, (const __half *)x, M, ln, epi)
                  : f32_linear_t<float>(ctx, w, (const float *)x, M, ln, epi);
}
