// Causal prefill attention on the tensor cores (tcgen05, accumulators in tensor memory), pipelined.
//
// Two persistent blocks per SM; each takes items (128-query tile, sequence, head) in turn, its copies and MMAs running on
// into the next item while the last one's output leaves.  Two warpgroups with fixed roles:
//   warp 0      copies: an item's Q tile, then the K and V tiles of its 128-key steps through tensor maps
//               (cp.async.bulk.tensor, 128-byte swizzle, zero fill past the last cached row) into two-stage
//               rings; no hand-written shared-memory stores anywhere
//   warp 1      MMA issue: S_t = Q K_t^T as soon as the softmax threads have S_{t-1} in their registers, then
//               O (+)= P_{t-1} V_{t-1} with P read from tensor memory (A operand) and V straight from its row-major tile
//               (B operand MN-major: no transposition)
//   warps 4..7  softmax: one thread per query row (= TMEM lane).  It takes the row's 128 scores once and keeps them in registers
//               from the maximum to the exponentials; p = exp2(s*scale - max) goes to tensor memory as packed fp16 when
//               the step before has finished with its own.  O stays in tensor memory over an item's steps and is
//               rescaled where a maximum has moved.
// A thread needs about 190 registers: the other warpgroup hands over its own (setmaxnreg: 40 + 208 of the 2 x 128 that the block
// was launched with).  What bounds it is the exponentials (16 per cycle and SM: 1024 of the 1800 cycles of a 128 x 128
// step) and the chain of a step that the other block's step has to cover: 125 cycles of TMEM loads, 250 of maxima, 1400 of
// exponentials, 300 of hand-overs.  Against one block per item, two threads per row, scores read twice, O folded into
// registers every step, 12 / 12 / 25 heads, us: 8 prompts of 1024 37.6 / 31.4 now, 32 of 512 49.7 / 37.6, 16 of 400 behind 100
// 59.1 / 45.1.  A reference that moves only past 2^8 saves another microsecond, and loses the exactness of the
// largest probabilities (error 2.51e-4 -> 2.55e-4): not taken.  A quarter of the exponentials as polynomials: 29.8 us for the 8 prompts
// of 1024, slower at every other size.  A single step in few blocks gains nothing (8 prompts of 128, 12 heads, the kernel alone: 5.9 / 6.1).
//
// TMEM (256 columns per block): S at columns 0..127, P (fp16 pairs) at 128..191, O at 192..255.
//
// Replaces flash_attention_v2 / flash_attn_v3.cu of the reference (compute_transformer.rs:597-816,
// cuda/flash_attn_v3.cu:29-283) for the model path, where q and the output are fp16.
//
// Every mbarrier wait is bounded: on expiry the block records a code in the device error word, all
// roles leave their loops, nothing more is stored (items it had finished are), the TMEM columns are freed and the kernel returns.
#include <cuda.h>

#include <algorithm>

#include "device_utils.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr float SCALE_LOG2E = 0.125f * 1.4426950408889634f;
constexpr float NEG_BIG = -1.0e30f;
enum : uint32_t { ERR_ATT_Q = 0x41, ERR_ATT_K, ERR_ATT_V, ERR_ATT_S, ERR_ATT_P, ERR_ATT_O, ERR_ATT_FREE, ERR_ATT_KE, ERR_ATT_VE, ERR_ATT_QE };
constexpr int TM_COLS = 256, TM_P = 128, TM_O = 192;
constexpr int KV_STAGES = 2;
constexpr int TILE = 16384;                 // 128 rows x 64 fp16
constexpr int SMEM_BYTES = (2 + 2 * KV_STAGES) * TILE + 1024; // Q of two items, K ring, V ring + alignment slack
constexpr int NTHREADS = 256, SOFTMAX = 128;

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&h);
}

struct Bars {
    uint64_t q_full[2], q_empty[2];
    uint64_t k_full[KV_STAGES], k_empty[KV_STAGES], v_full[KV_STAGES], v_empty[KV_STAGES];
    uint64_t s_full, s_free, p_full, o_full; // one phase per step
};

__global__ void __launch_bounds__(NTHREADS, 2)
prefill_attn_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v, int H, int pairs, int cap, int S, int past,
                       __half *__restrict__ out, int ldo, uint32_t *__restrict__ dev_err) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) Bars bars;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;

    // Items are (query tile, sequence, head), those with the most key tiles first; a block's n-th is dealt out forwards and
    // backwards in turn, so that blocks come out even.
    const int q_tiles = (S + 127) / 128, n_items = q_tiles * pairs;
    struct Item {
        int qt, bh, kv_end, n_tiles;
    };
    auto item_at = [&](int n, Item &it) {
        const int i = n * gridDim.x + ((n & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
        if (i >= n_items) return false;
        it.qt = q_tiles - 1 - i / pairs;
        it.bh = i % pairs;
        it.kv_end = min(past + min(S, it.qt * 128 + 128), cap); // keys this tile's queries can see
        it.n_tiles = (it.kv_end + 127) / 128;
        return true;
    };
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t base = (tc::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t sQ = base, sK = base + 2 * TILE, sV = base + TILE * (2 + KV_STAGES);
    auto bar = [&](const uint64_t &x) { return tc::smem_u32(&x); };

    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(bar(bars.q_full[i]), 1);
            tc::mbar_init(bar(bars.q_empty[i]), 1);
        }
        for (int i = 0; i < KV_STAGES; ++i) {
            tc::mbar_init(bar(bars.k_full[i]), 1);
            tc::mbar_init(bar(bars.k_empty[i]), 1);
            tc::mbar_init(bar(bars.v_full[i]), 1);
            tc::mbar_init(bar(bars.v_empty[i]), 1);
        }
        tc::mbar_init(bar(bars.s_full), 1);
        tc::mbar_init(bar(bars.s_free), SOFTMAX / 32); // every softmax warp
        tc::mbar_init(bar(bars.p_full), SOFTMAX / 32);
        tc::mbar_init(bar(bars.o_full), 1);
        tc::fence_mbar_init();
    }
    if (warp == 0) {
        tc::prefetch_tmap(&tm_q);
        tc::prefetch_tmap(&tm_k);
        tc::prefetch_tmap(&tm_v);
    }
    if (warp == 1) tc::tmem_alloc(tc::smem_u32(&tmem_slot), TM_COLS);
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(&tmem_slot);

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        Item it;
        int t = 0; // step over all items
        if (warp == 0) {
            // ---- copies (one elected lane issues; the warp stays converged on the waits) ----
            bool ok = true;
            for (int n = 0; ok && item_at(n, it); ++n) {
                if (n >= 2) ok = tc::mbar_wait(bar(bars.q_empty[n & 1]), ((n >> 1) - 1) & 1, &abort_flag, dev_err, ERR_ATT_QE);
                if (!ok) break;
                if (tc::elect_one()) {
                    tc::mbar_expect_tx(bar(bars.q_full[n & 1]), TILE);
                    tc::tma_load_2d(sQ + (n & 1) * TILE, &tm_q, it.bh % H * 64, it.bh / H * S + it.qt * 128, bar(bars.q_full[n & 1]));
                }
                for (int j = 0; j < it.n_tiles; ++j, ++t) {
                    const int st = t % KV_STAGES, u = t / KV_STAGES;
                    if (t >= KV_STAGES) ok = tc::mbar_wait(bar(bars.k_empty[st]), (u - 1) & 1, &abort_flag, dev_err, ERR_ATT_KE);
                    if (!ok) break;
                    if (tc::elect_one()) {
                        tc::mbar_expect_tx(bar(bars.k_full[st]), TILE);
                        tc::tma_load_3d(sK + st * TILE, &tm_k, 0, j * 128, it.bh, bar(bars.k_full[st]));
                    }
                    if (t >= KV_STAGES) ok = tc::mbar_wait(bar(bars.v_empty[st]), (u - 1) & 1, &abort_flag, dev_err, ERR_ATT_VE);
                    if (!ok) break;
                    if (tc::elect_one()) {
                        tc::mbar_expect_tx(bar(bars.v_full[st]), TILE);
                        tc::tma_load_3d(sV + st * TILE, &tm_v, 0, j * 128, it.bh, bar(bars.v_full[st]));
                    }
                }
            }
        } else if (warp == 1) {
            // ---- MMA issue: S_t once S_{t-1} has been read and K_t is there, O (+)= P_{t-1} V_{t-1} once P_{t-1} is written ----
            constexpr uint32_t idesc_s = tc::umma_idesc_f16(128, 128);
            constexpr uint32_t idesc_o = tc::umma_idesc_f16_bmn(128, 64);
            auto output = [&](int tp, bool first) {
                const int st = tp % KV_STAGES, u = tp / KV_STAGES;
                if (!tc::mbar_wait(bar(bars.p_full), tp & 1, &abort_flag, dev_err, ERR_ATT_P) ||
                    !tc::mbar_wait(bar(bars.v_full[st]), u & 1, &abort_flag, dev_err, ERR_ATT_V))
                    return false;
                tc::tc_fence_after_sync();
                if (tc::elect_one()) {
                    const uint64_t dv = tc::umma_desc_sw128_mn64(sV + st * TILE);
#pragma unroll
                    for (int k = 0; k < 8; ++k) // 16 keys per MMA: 8 TMEM columns of P, 2048 bytes of V
                        tc::umma_f16_ts(tmem_base + TM_O, tmem_base + TM_P + 8 * k, dv + (uint64_t)(k * (2048 >> 4)), idesc_o, !first || k != 0);
                    tc::umma_commit(bar(bars.o_full));
                    tc::umma_commit(bar(bars.v_empty[st]));
                }
                __syncwarp();
                return true;
            };
            bool ok = true, first = true; // whether step t - 1 is its item's first
            for (int n = 0; ok && item_at(n, it); ++n) {
                ok = tc::mbar_wait(bar(bars.q_full[n & 1]), (n >> 1) & 1, &abort_flag, dev_err, ERR_ATT_Q);
                const uint64_t dq = tc::umma_desc_sw128(sQ + (n & 1) * TILE);
                for (int j = 0; ok && j < it.n_tiles; ++j, ++t) {
                    const int st = t % KV_STAGES, u = t / KV_STAGES;
                    if (t >= 1) ok = tc::mbar_wait(bar(bars.s_free), (t - 1) & 1, &abort_flag, dev_err, ERR_ATT_FREE);
                    if (ok) ok = tc::mbar_wait(bar(bars.k_full[st]), u & 1, &abort_flag, dev_err, ERR_ATT_K);
                    if (!ok) break;
                    tc::tc_fence_after_sync();
                    if (tc::elect_one()) {
                        const uint64_t dk = tc::umma_desc_sw128(sK + st * TILE);
#pragma unroll
                        for (int k = 0; k < 4; ++k) tc::umma_f16_ss(tmem_base, dq + 2 * k, dk + 2 * k, idesc_s, k != 0);
                        tc::umma_commit(bar(bars.s_full));
                        tc::umma_commit(bar(bars.k_empty[st]));
                        if (j + 1 == it.n_tiles) tc::umma_commit(bar(bars.q_empty[n & 1]));
                    }
                    __syncwarp();
                    if (t >= 1) ok = output(t - 1, first);
                    first = j == 0;
                }
            }
            if (ok) output(t - 1, first);
        }
    } else {
        // ---- softmax: one thread per query row (= TMEM lane) ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int quad = warp & 3, row = quad * 32 + (tid & 31);
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
        float m = NEG_BIG;
        float2 l2[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        uint4 *dst = nullptr; // output row of the item before (null: none, or past the sequence)
        // The finished O of an item leaves (its last MMA has completed).
        auto finish = [&]() {
            const float inv = 1.0f / ((l2[0].x + l2[0].y) + (l2[1].x + l2[1].y));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint32_t o[32];
                tc::tmem_ld_x32(lane_base + TM_O + 32 * i, o);
                if (dst)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            w[e] = pack_half2(__uint_as_float(o[8 * c + 2 * e]) * inv, __uint_as_float(o[8 * c + 2 * e + 1]) * inv);
                        dst[4 * i + c] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
            }
        };
        Item it;
        int t = 0;
        bool ok = true;
        for (int n = 0; ok && item_at(n, it); ++n) {
            // Rows past the sequence are worked out like the others (their queries are the next sequence's, or zeros) and not stored.
            const int s_row = it.qt * 128 + row, a_pos = past + s_row; // absolute position of this thread's query
            const int warp_row = it.qt * 128 + quad * 32, warp_first = past + warp_row; // last key that all rows of the warp see
            const int warp_last = warp_row < S ? min(warp_first + 31, it.kv_end - 1) : -1; // last key that any of them sees
            for (int j = 0; j < it.n_tiles; ++j, ++t) {
                const int j0 = j * 128;
                ok = tc::mbar_wait(bar(bars.s_full), t & 1, &abort_flag, dev_err, ERR_ATT_S);
                if (!ok) break;
                tc::tc_fence_after_sync();
                uint32_t v[2][64];
                tc::tmem_ld_x64(lane_base, v[0]);
                tc::tmem_ld_x64(lane_base + 64, v[1]);
                tc::tc_fence_before_sync();
                __syncwarp();
                if ((tid & 31) == 0) tc::mbar_arrive(bar(bars.s_free)); // S_{t+1} may take their place
                // the row may attend to keys up to a_pos.  Only the tile on the diagonal needs the mask: masked scores lie so far below any other that their exponentials are zero.
                float mx[4] = {NEG_BIG, NEG_BIG, NEG_BIG, NEG_BIG}; // four independent chains
                auto maxima = [&](int c) {
#pragma unroll
                    for (int e = 32 * c; e < 32 * c + 32; e += 8)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            mx[i] = tc::fmax3(mx[i], __uint_as_float(v[e >> 6][(e & 63) + 2 * i]), __uint_as_float(v[e >> 6][(e & 63) + 2 * i + 1]));
                };
                if (j0 + 127 <= warp_first) { // (uniform)
#pragma unroll
                    for (int c = 0; c < 4; ++c) maxima(c);
                } else {
                    const int nvalid = a_pos - j0 + 1;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (j0 + 32 * c > warp_last) break; // (uniform) nothing that a row of the warp sees
                        if (j0 + 32 * c + 31 > warp_first)
#pragma unroll
                            for (int e = 0; e < 32; ++e)
                                if (32 * c + e >= nvalid) v[c >> 1][(c & 1) * 32 + e] = __float_as_uint(NEG_BIG);
                        maxima(c);
                    }
                }
                const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * SCALE_LOG2E;
                const float next = j == 0 ? top : fmaxf(m, top), corr = tc::ex2_approx(m - next);
                const bool moved = __any_sync(0xffffffffu, next > m);
                // p = 2^(s*scale - maximum), in the scores' registers; the MMAs of the step before run meanwhile
                const float2 sc2 = make_float2(SCALE_LOG2E, SCALE_LOG2E), nm2 = make_float2(-next, -next);
                float2 ls[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
                uint32_t o[4][16];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (j0 + 32 * c > warp_last) { // (uniform)
#pragma unroll
                        for (int e = 0; e < 16; ++e) o[c][e] = 0u;
                    } else {
#pragma unroll
                        for (int e = 0; e < 32; e += 2) {
                            const float2 x = __ffma2_rn(make_float2(__uint_as_float(v[c >> 1][(c & 1) * 32 + e]), __uint_as_float(v[c >> 1][(c & 1) * 32 + e + 1])), sc2, nm2);
                            const float2 p = make_float2(tc::ex2_approx(x.x), tc::ex2_approx(x.y));
                            ls[(e >> 1) & 1] = __fadd2_rn(ls[(e >> 1) & 1], p);
                            o[c][e >> 1] = pack_half2(p.x, p.y);
                        }
                    }
                }
                if (t >= 1) { // P's place is free and O complete
                    ok = tc::mbar_wait(bar(bars.o_full), (t - 1) & 1, &abort_flag, dev_err, ERR_ATT_O);
                    if (!ok) break;
                    tc::tc_fence_after_sync();
                }
                if (j == 0) {
                    if (n) finish();
                    dst = s_row < S ? reinterpret_cast<uint4 *>(out + ((size_t)(it.bh / H) * S + s_row) * ldo + it.bh % H * 64) : nullptr;
                    l2[0] = ls[0];
                    l2[1] = ls[1];
                } else {
                    if (moved) {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            uint32_t w[32];
                            tc::tmem_ld_x32(lane_base + TM_O + 32 * i, w);
#pragma unroll
                            for (int e = 0; e < 32; ++e) w[e] = __float_as_uint(__uint_as_float(w[e]) * corr);
                            tc::tmem_st_x32(lane_base + TM_O + 32 * i, w);
                            l2[i] = make_float2(l2[i].x * corr, l2[i].y * corr);
                        }
                    }
                    l2[0] = __fadd2_rn(l2[0], ls[0]);
                    l2[1] = __fadd2_rn(l2[1], ls[1]);
                }
                m = next;
#pragma unroll
                for (int c = 0; c < 4; ++c) tc::tmem_st_x16(lane_base + TM_P + 16 * c, o[c]);
                tc::tmem_st_wait();
                tc::tc_fence_before_sync();
                __syncwarp();
                if ((tid & 31) == 0) tc::mbar_arrive(bar(bars.p_full));
            }
        }
        if (ok) ok = tc::mbar_wait(bar(bars.o_full), (t - 1) & 1, &abort_flag, dev_err, ERR_ATT_O);
        if (ok) { // (warp-uniform)
            tc::tc_fence_after_sync();
            finish();
        }
    }

    // ---- teardown (also the path taken after a wait gave up) ----
    if (abort_flag && warp == 0) { // let copies still in flight land before the block's memory is released
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem_base, TM_COLS);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

}  // namespace

// q, out fp16; rows of q / out are ldq / H*64 halves apart and must be 16-byte aligned, as must q, kc and vc.
int launch_prefill_attention_tc(b200nn_ctx *ctx, const __half *q, int ldq, const __half *kc, const __half *vc, int B, int H,
                                int cap, int S, int past, __half *out) {
    if (!ctx->encode_tiled) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is unavailable");
    if (((uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc | (uintptr_t)out) & 15 || (ldq & 7))
        return set_error(ctx, B200NN_ERR_ARG, "prefill attention: q, K, V and out must be 16-byte aligned, rows of q a multiple of 8 halves");
    static bool attr_done[16] = {};
    if (!attr_done[ctx->device & 15]) {
        CK(ctx, cudaFuncSetAttribute(prefill_attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        prefer_max_smem(prefill_attn_tc_kernel);
        attr_done[ctx->device & 15] = true;
    }
    const EncodeTiledFn encode = (EncodeTiledFn)ctx->encode_tiled;
    CUtensorMap tq, tk, tv;
    const cuuint32_t ones[3] = {1, 1, 1};
    {   // queries: [B*S rows][H*64] fp16, rows ldq halves apart; one box = 128 rows of one head
        cuuint64_t dim[2] = {(cuuint64_t)H * 64, (cuuint64_t)B * S};
        cuuint64_t stride[1] = {(cuuint64_t)ldq * sizeof(__half)};
        cuuint32_t box[2] = {64, 128};
        CUresult r = encode(&tq, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void *)q, dim, stride, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return set_error(ctx, B200NN_ERR_CUDA, "cuTensorMapEncodeTiled (q) failed: " + std::to_string((int)r));
    }
    // K and V caches: [B*H][cap rows][64] fp16; the row extent is the number of rows written so far, so
    // that a box reaching past it is zero-filled instead of reading rows nothing has written
    const cuuint64_t rows = (cuuint64_t)std::min(past + S, cap);
    cuuint64_t dim[3] = {64, rows, (cuuint64_t)B * H};
    cuuint64_t stride[2] = {64 * sizeof(__half), (cuuint64_t)cap * 64 * sizeof(__half)};
    cuuint32_t box[3] = {64, 128, 1};
    for (int which = 0; which < 2; ++which) {
        CUresult r = encode(which ? &tv : &tk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void *)(which ? vc : kc), dim, stride, box, ones,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return set_error(ctx, B200NN_ERR_CUDA, "cuTensorMapEncodeTiled (K/V) failed: " + std::to_string((int)r));
    }
    const long long items = (long long)B * H * ((S + 127) / 128);
    if (B > 65535 || (S + 127) / 128 > 65535 || items > 0x3fffffff)
        return set_error(ctx, B200NN_ERR_SHAPE, "prefill attention: more than 65535 sequences or query tiles");
    const int grid = (int)std::min<long long>(items, 2 * ctx->sm_count);
    prefill_attn_tc_kernel<<<grid, NTHREADS, SMEM_BYTES, ctx->stream>>>(tq, tk, tv, H, B * H, cap, S, past, out, H * 64, ctx->dev_err);
    CK_LAUNCH(ctx, "prefill_attn_tc_kernel");
    return B200NN_OK;
}
