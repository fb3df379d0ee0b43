// Group-wise int4 weight-only Linear on CUDA cores.
//
//   int4_gemv_kernel   few input rows (decode of one or two sequences): HBM-bound streaming of the
//                      tiled nibbles with 128-bit coalesced loads (three K blocks per thread in
//                      flight, the first ones issued before the wait on the preceding kernel:
//                      weights do not depend on it), in-register dequantisation, f32 accumulation.
//                      K is split inside a block and up to eight ways across the blocks of
//                      a thread-block cluster; the blocks store their partial sums into the
//                      shared memory of the cluster's first block, which adds them (fixed order, no
//                      global scratch, no atomics) and runs the fused bias / activation /
//                      residual / KV-cache epilogue.  A LayerNorm of the input rows can ride along.
//   int4_naive_kernel  any K%8==0 and any group size, reference layout, one thread per output as
//                      crates/kernel/gpu-kernel-compute/src/compute_gemm.rs:2849-2910 does.
//
// Both compute y[m,n] = sum_k x[m,k] * (nibble(k,n)-8) * scale[k/group,n] (+ bias[n]).
#include "device_utils.cuh"

static constexpr int GEMV_THREADS = 512;
// K blocks of a thread in flight: as many as the 64 registers of two blocks per SM hold beside the row sums and a LayerNorm's
// values; three where the registers of a whole SM are there for one block.
template <int MT, bool LN, int PER_SM>
constexpr int gemv_ahead = MT == 1 || (MT == 2 && !LN) || PER_SM == 1 ? 3 : 2;

template <int MT>
__device__ __forceinline__ void gemv_block_fma(const uint4 &wa, const uint4 &wb, float s, const float *xb, int len,
                                               float (&acc)[MT]) {
    const uint32_t w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
    float part[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) part[m] = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        __half2 q[4];
        unpack8_int4(w[j], q);
        const float2 f0 = __half22float2(q[0]), f1 = __half22float2(q[1]);
        const float2 f2 = __half22float2(q[2]), f3 = __half22float2(q[3]);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float4 xa = *reinterpret_cast<const float4 *>(xb + m * len + 8 * j);
            const float4 xc = *reinterpret_cast<const float4 *>(xb + m * len + 8 * j + 4);
            float p = part[m];
            p = fmaf(xa.x, f0.x, p); p = fmaf(xa.y, f0.y, p);
            p = fmaf(xa.z, f1.x, p); p = fmaf(xa.w, f1.y, p);
            p = fmaf(xc.x, f2.x, p); p = fmaf(xc.y, f2.y, p);
            p = fmaf(xc.z, f3.x, p); p = fmaf(xc.w, f3.y, p);
            part[m] = p;
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = fmaf(s, part[m], acc[m]);
}

// grid (weight rows / RW, splits), cluster (1, splits, 1): the blocks of a cluster share RW rows of the weight.  A thread
// has one row and every SLICES-th K block of its block's range.  RW 128: four slices.  RW 32: sixteen, for weights of
// few rows, so that a thread has two or three K blocks, all of them requested before the wait, and most weights need no
// second block per tile.  LN: the rows' LayerNorm is taken here; one f32 row has one kernel for both and asks `ln.g`, two have
// the values that the LayerNorm holds in shared memory and a kernel of their own for it (in registers they spilled: two
// sequences of GPT-2 Small, 64 tokens after a prompt of 64: 23.6 -> 20.4 ms).
template <int MT, int RW, bool LN, int PER_SM, typename XT>
__global__ void __launch_bounds__(GEMV_THREADS, PER_SM)
int4_gemv_kernel(const uint4 *__restrict__ tiles, const __half *__restrict__ scales, Fresh<XT> x,
                 int m_valid, int m0, int K, int N, int k_blocks, int n_pad, int group, int kb_per_split,
                 NormIn ln, Epilogue epi) {
    constexpr int SLICES = GEMV_THREADS / RW, AHEAD = gemv_ahead<MT, LN, PER_SM>;
    extern __shared__ float smem_f[];
    const int split = blockIdx.y, splits = gridDim.y;
    const int tid = threadIdx.x, r = tid % RW, slice = tid / RW;
    const int n = blockIdx.x * RW + r, tile_row = n & 127;
    const int kb0 = split * kb_per_split;
    const int kb1 = min(kb0 + kb_per_split, k_blocks);
    const int len = kb_per_split * 64;
    float *xs = smem_f;                        // [MT][len] activations of this block's K range
    float *red = smem_f + MT * len;            // [SLICES][MT][RW] slice sums
    float *part = red + SLICES * MT * RW;      // [splits][MT][RW] partial tiles, in the cluster's first block
    float *held = part + splits * MT * RW;     // two rows with a LayerNorm: [MT + 2][K]
    pdl_trigger();
    if (splits > 1) cluster_arrive(); // waited for before the first store into another block

    // weights and scales of this thread's first K blocks: issued before the wait on the
    // previous kernel (they are constants), so that their DRAM latency overlaps its tail
    const uint4 *tile0 = tiles + (size_t)(n >> 7) * k_blocks * (TILE_BYTES / 16) + tile_row;
    uint4 wa[AHEAD], wb[AHEAD];
    float sc[AHEAD];
    auto load_block = [&](int i, int kb) {
        if (kb >= kb1) return;
        const uint4 *tp = tile0 + (size_t)kb * (TILE_BYTES / 16);
        wa[i] = __ldg(tp);
        wb[i] = __ldg(tp + 128);
        sc[i] = __half2float(scales[(size_t)((kb * 64) / group) * n_pad + n]);
    };
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) load_block(i, kb0 + slice + i * SLICES);

    if constexpr (LN) {
        if (MT > 1 || ln.g) norm_rows_to_smem<MT, GEMV_THREADS, (MT > 1)>(ln, x, m_valid, K, kb0 * 64, (kb1 - kb0) * 64, len, xs, red, held);
    }
    if (!LN || (MT == 1 && !ln.g)) {
        pdl_wait();
        rows_to_smem<MT, GEMV_THREADS>(x, m_valid, K, kb0 * 64, (kb1 - kb0) * 64, len, xs);
    }
    __syncthreads();

    float acc[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = 0.0f;
    for (int kb = kb0 + slice; kb < kb1; kb += AHEAD * SLICES) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int k = kb + i * SLICES;
            if (k < kb1) gemv_block_fma<MT>(wa[i], wb[i], sc[i], xs + (k - kb0) * 64, len, acc);
            load_block(i, k + AHEAD * SLICES);
        }
    }

#pragma unroll
    for (int m = 0; m < MT; ++m) red[(slice * MT + m) * RW + r] = acc[m];
    __syncthreads();
    float t = 0.0f; // thread m * RW + r: feature r of row m (MT * RW <= GEMV_THREADS)
    const int m = slice;
    if (m < MT)
#pragma unroll
        for (int sl = 0; sl < SLICES; ++sl) t += red[(sl * MT + m) * RW + r];
    if (splits > 1) {
        cluster_wait();
        if (m < MT) st_cluster(&part[(split * MT + m) * RW + r], 0, t);
        cluster_arrive();
        cluster_wait(); // every block's partial tile is in the first block
        if (split != 0) return;
        t = 0.0f;
        if (m < MT)
            for (int sp = 0; sp < splits; ++sp) // fixed order: the result does not depend on timing
                t += part[(sp * MT + m) * RW + r];
    }
    if (m < min(MT, m_valid)) { // RW / 32 warps per row: 32 consecutive features each
        if (n < N) epi_apply(epi, m0 + m, n, t);
        if (epi.amax_val) epi_argmax1(epi, m0 + m, n, t + (epi.bias && n < N ? epi.bias[n] : 0.0f), n < N);
    }
}

template <typename XT>
__global__ void int4_naive_kernel(const uint32_t *__restrict__ packed, const float *__restrict__ scales,
                                  const XT *__restrict__ x, int M, int N, int K, int group, Epilogue epi) {
    size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (size_t)M * N) return;
    int row = id / N, col = id % N;
    float acc = 0.0f;
    for (int kp = 0; kp < K / 8; ++kp) {
        uint32_t w = packed[(size_t)kp * N + col];
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
            int ki = kp * 8 + bit;
            int q = (int)((w >> (bit * 4)) & 0xFu) - 8;
            float wf = (float)q * scales[(size_t)(ki / group) * N + col];
            acc = fmaf(load_as_float<XT>(x, (size_t)row * K + ki), wf, acc);
        }
    }
    epi_apply(epi, row, col, acc);
}

int launch_int4_naive(b200nn_ctx *ctx, const Int4Weight &w, const void *x, bool x_half, int M, const Epilogue &epi) {
    if (M <= 0) return B200NN_OK;
    if (!w.ref_packed) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "int4 weight has no reference-layout copy");
    size_t total = (size_t)M * w.N;
    int grid = (int)((total + 255) / 256);
    PREFER_SMEM_ONCE(int4_naive_kernel<__half>);
    PREFER_SMEM_ONCE(int4_naive_kernel<float>);
    if (x_half)
        int4_naive_kernel<__half><<<grid, 256, 0, ctx->stream>>>((const uint32_t *)w.ref_packed->p,
                                                                 (const float *)w.ref_scales->p, (const __half *)x, M,
                                                                 w.N, w.K, w.group, epi);
    else
        int4_naive_kernel<float><<<grid, 256, 0, ctx->stream>>>((const uint32_t *)w.ref_packed->p,
                                                                (const float *)w.ref_scales->p, (const float *)x, M,
                                                                w.N, w.K, w.group, epi);
    CK_LAUNCH(ctx, "int4_naive_kernel");
    return B200NN_OK;
}

template <int MT, int RW, bool LN, int PER_SM, typename XT>
static int gemv_launch(b200nn_ctx *ctx, const Int4Weight &w, const XT *x, int m_valid, int m0, const NormIn &ln, const Epilogue &epi) {
    constexpr int SLICES = GEMV_THREADS / RW;
    constexpr size_t SMEM_MAX = 216 * 1024;
    // K split across a cluster of up to eight blocks so that about one block per SM is resident; the sixteen slices of
    // a narrow block have a K block each at least
    const int tiles = (w.N + RW - 1) / RW;
    int splits = RW == 32 ? ctx->sm_count / tiles : (ctx->sm_count + tiles - 1) / tiles;
    splits = std::max(1, std::min(splits, 8));
    splits = std::min(splits, std::max(1, w.k_blocks / SLICES));
    const int per = (w.k_blocks + splits - 1) / splits;
    splits = (w.k_blocks + per - 1) / per;
    const size_t smem = ((size_t)MT * per * 64 + (size_t)(SLICES + splits) * MT * RW + (LN && MT > 1 ? (MT + 2) * w.K : 0)) * sizeof(float);
    auto kern = int4_gemv_kernel<MT, RW, LN, PER_SM, XT>;
    static bool attr_done[16] = {}; // function attributes are per device
    if (!attr_done[ctx->device & 15]) {
        CK(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX));
        prefer_max_smem(kern);
        attr_done[ctx->device & 15] = true;
    }
    if (smem > SMEM_MAX) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "int4 GEMV: K too large for one cluster");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, splits);
    cfg.blockDim = dim3(GEMV_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = splits;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = ctx->pdl ? attr : attr + 1;
    cfg.numAttrs = (ctx->pdl ? 1 : 0) + (splits > 1 ? 1 : 0);
    CK(ctx, cudaLaunchKernelEx(&cfg, kern, (const uint4 *)w.tiled->p, (const __half *)w.scales_h->p, x, m_valid, m0, w.K,
                               w.N, w.k_blocks, w.n_pad, w.group, per, ln, epi));
    CK_LAUNCH(ctx, "int4_gemv_kernel");
    return B200NN_OK;
}
template <int MT, bool LN, typename XT>
static int gemv_chunk(b200nn_ctx *ctx, const Int4Weight &w, const XT *x, int m_valid, int m0, const NormIn &ln, const Epilogue &epi) {
    // 32 rows a block while the blocks stay under two per SM and the activations of a block's K range small (an output
    // matrix has its blocks in 128 rows: ten blocks per SM would each pay for the start)
    const int tiles = (w.N + 31) / 32, splits = std::max(1, std::min(8, ctx->sm_count / tiles)), per = (w.k_blocks + splits - 1) / splits;
    const bool narrow = tiles <= 2 * ctx->sm_count && (size_t)MT * per * 64 * sizeof(float) <= 96 * 1024;
    if constexpr (MT == 1 && sizeof(XT) == 4) {
        return narrow ? gemv_launch<1, 32, true, 2, XT>(ctx, w, x, m_valid, m0, ln, epi) : gemv_launch<1, 128, true, 2, XT>(ctx, w, x, m_valid, m0, ln, epi);
    } else if constexpr (LN) { // K is short, N a few times K
        return gemv_launch<MT, 32, true, 2, XT>(ctx, w, x, m_valid, m0, ln, epi);
    } else {
        if constexpr (MT == 4) // a block per SM at most: its registers hold three K blocks (6400 x 1600, four rows: 13.3 -> 9.8 us)
            if (narrow && tiles <= ctx->sm_count) return gemv_launch<4, 32, false, 1, XT>(ctx, w, x, m_valid, m0, ln, epi);
        return narrow ? gemv_launch<MT, 32, false, 2, XT>(ctx, w, x, m_valid, m0, ln, epi) : gemv_launch<MT, 128, false, 2, XT>(ctx, w, x, m_valid, m0, ln, epi);
    }
}

template <bool LN, typename XT>
static int gemv_all(b200nn_ctx *ctx, const Int4Weight &w, const XT *x, int M, const NormIn &ln, const Epilogue &epi) {
    int m0 = 0;
    while (m0 < M) {
        int left = M - m0;
        const XT *xp = x + (size_t)m0 * w.K;
        if (left >= 4) {
            TRY((gemv_chunk<4, false, XT>(ctx, w, xp, 4, m0, ln, epi)));
            m0 += 4;
        } else if (left >= 2) {
            TRY((gemv_chunk<2, LN, XT>(ctx, w, xp, 2, m0, ln, epi)));
            m0 += 2;
        } else {
            TRY((gemv_chunk<1, LN, XT>(ctx, w, xp, 1, m0, ln, epi)));
            m0 += 1;
        }
    }
    return B200NN_OK;
}

// (four rows at a time and a LayerNorm do not fit the registers beside the weights in flight)
bool int4_linear_takes_norm(const Int4Weight &w, int M) { return w.fast && M >= 1 && M <= 2 && w.K <= NORM_IN_MAX; }

int launch_int4_gemv(b200nn_ctx *ctx, const Int4Weight &w, const void *x, bool x_half, int M, const Epilogue &epi, const NormIn &ln) {
    if (M <= 0) return B200NN_OK;
    if (ln.g && (x_half || !int4_linear_takes_norm(w, M)))
        return set_error(ctx, B200NN_ERR_UNSUPPORTED, "int4 Linear: only the GEMV of few rows takes a LayerNorm with its input");
    if (epi.ln_stats || epi.mode == EPI_RESID_LN) { // folded LayerNorms exist in the tensor-core GEMM's epilogue only
        if (!(w.fast && M > ctx->gemv_max_rows && x_half && int4_gemm_tc_supported(w, M)) || int4_via_f16_supported(ctx, w, M))
            return set_error(ctx, B200NN_ERR_UNSUPPORTED, "folded LayerNorm: this Linear does not run on the tensor-core GEMM");
        return launch_int4_gemm_tc(ctx, w, (const __half *)x, M, epi);
    }
    if (!w.fast) return launch_int4_naive(ctx, w, x, x_half, M, epi);
    if (x_half) return gemv_all<false, __half>(ctx, w, (const __half *)x, M, ln, epi);
    return ln.g ? gemv_all<true, float>(ctx, w, (const float *)x, M, ln, epi) : gemv_all<false, float>(ctx, w, (const float *)x, M, ln, epi);
}

int launch_int4_linear(b200nn_ctx *ctx, const Int4Weight &w, const void *x, bool x_half, int M, const Epilogue &epi, const NormIn &ln) {
    if (M <= 0) return B200NN_OK;
    if (ln.g) return launch_int4_gemv(ctx, w, x, x_half, M, epi, ln);
    if (epi.ln_stats || epi.mode == EPI_RESID_LN) { // folded LayerNorms exist in the tensor-core GEMM's epilogue only
        if (!(w.fast && M > ctx->gemv_max_rows && x_half && int4_gemm_tc_supported(w, M)) || int4_via_f16_supported(ctx, w, M))
            return set_error(ctx, B200NN_ERR_UNSUPPORTED, "folded LayerNorm: this Linear does not run on the tensor-core GEMM");
        return launch_int4_gemm_tc(ctx, w, (const __half *)x, M, epi);
    }
    if (!w.fast) return launch_int4_naive(ctx, w, x, x_half, M, epi);
    // a prefill pass with at least two 256-row tiles per SM: dequantise once, persistent fp16 GEMM
    if (x_half && !((uintptr_t)x & 15) && int4_via_f16_supported(ctx, w, M))
        return launch_int4_via_f16(ctx, w, (const __half *)x, M, epi);
    if (M > ctx->gemv_max_rows && x_half && int4_gemm_tc_supported(w, M))
        return launch_int4_gemm_tc(ctx, w, (const __half *)x, M, epi);
    return launch_int4_gemv(ctx, w, x, x_half, M, epi);
}
