// Device-side helpers shared by the kernels: activations, the Linear epilogue, reductions.
#pragma once
#include "common.h"

// Programmatic dependent launch: wait until the preceding kernel on the stream has completed and
// its writes are visible (a no-op when the kernel was not launched as a programmatic dependent),
// and allow the following kernel to begin launching.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ float gelu_tanh_f(float x) {
    // x*0.5*(1+tanh(sqrt(2/pi)*(x+0.044715x^3))): the GPT-2 form used by the reference's CPU model
    // (crates/test/gpu-test-harness/src/tests_inference.rs:3680-3685).
    // 0.5*(1+tanh(u)) == 1/(1+exp(-2u)): one exponential and one division instead of tanhf's ~25
    // instructions (the GELU of a 256x128 tile was two thirds of the FC epilogue's time).  u is
    // clamped where the result is already zero to within 1e-30 so that the exponential stays finite.
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    float inner = fmaxf(k0 * (x + k1 * x * x * x), -40.0f);
    return __fdividef(x, 1.0f + __expf(-2.0f * inner));
}

__device__ __forceinline__ float gelu_sigmoid_f(float x) {
    // x*sigmoid(1.702x): crates/kernel/gpu-kernel-compute/src/compute_transformer.rs:1486-1504.
    return x / (1.0f + __expf(-1.702f * x));
}

__device__ __forceinline__ float apply_act(float v, int act) {
    switch (act) {
        case B200NN_ACT_GELU_TANH: return gelu_tanh_f(v);
        case B200NN_ACT_GELU_SIGMOID: return gelu_sigmoid_f(v);
        case B200NN_ACT_RELU: return fmaxf(v, 0.0f);
        case B200NN_ACT_SILU: return v / (1.0f + __expf(-v));
        case B200NN_ACT_SIGMOID: return 1.0f / (1.0f + __expf(-v));
        default: return v;
    }
}

__device__ __forceinline__ float4 f4_add(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t pack_f16x2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// A value that an earlier kernel of the chain wrote, read after pdl_wait: from L2.  The block may have been resident while
// that kernel ran on the same SM, so a line that came into L1 since this kernel's start (or through the read-only
// path, which a plain load from a const __restrict__ pointer takes) can be older than the wait: the second of four f32 rows
// got its MLP from the residual stream without the attention's sum.
// (volatile: it stays behind the wait, and in the order of the source, so values that should be in flight together are
// loaded before the first of them is used)
__device__ __forceinline__ int load_fresh_int(const void *p) {
    int v;
    asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float load_fresh(const float *p, size_t i) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p + i));
    return v;
}
__device__ __forceinline__ float load_fresh(const __half *p, size_t i) {
    unsigned short v;
    asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(v) : "l"(p + i));
    return __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ uint32_t load_fresh(const uint32_t *p, size_t i) { return (uint32_t)load_fresh_int(p + i); }
__device__ __forceinline__ int load_fresh(const int *p, size_t i) { return load_fresh_int(p + i); }
__device__ __forceinline__ float2 load_fresh(const float2 *p, size_t i) { return __ldcg(p + i); }
__device__ __forceinline__ float4 load_fresh(const float4 *p, size_t i) { return __ldcg(p + i); }
__device__ __forceinline__ uint4 load_fresh(const uint4 *p, size_t i) { return __ldcg(p + i); }
__device__ __forceinline__ float4 load_fresh4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }
// The parameter through which a kernel launched with launch_pdl takes an array that earlier kernels of the chain write:
// it has no plain reads.  (p is for copies that go past L1 anyway: cp.async.cg, bulk copies.)
template <typename T>
struct Fresh {
    const T *p;
    __host__ __device__ Fresh(const T *q) : p(q) {}
    __device__ __forceinline__ explicit operator bool() const { return p != nullptr; }
    __device__ __forceinline__ Fresh operator+(size_t n) const { return Fresh(p + n); }
    __device__ __forceinline__ auto operator[](size_t i) const { return load_fresh(p, i); }
    __device__ __forceinline__ float4 four(size_t i) const { return load_fresh4(p + i); } // floats i .. i+3, i a multiple of 4
};
__device__ __forceinline__ int row_pos(const RowMap &r, int m) { return load_fresh_int(r.pos + (size_t)m * r.pos_stride); }
__device__ __forceinline__ int row_slot(const RowMap &r, int m) { return r.slot ? r.slot[m] : m; }

// Consumes one finished output value v (bias already added) for row m (token), column n (feature).
// B16: with the bfloat16 Linears' additions (bfloat16 output, EPI_GLU, EPI_ROPE, row_scale); kernels that never see
// them leave the code out (it costs the int4 GEMM's epilogue 5 % of a decode step's Linears).
template <bool B16 = false>
__device__ __forceinline__ void epi_store(const Epilogue &e, int m, int n, float v) {
    if (e.no_store) return;
    if (e.mode == EPI_RESID) {
        size_t i = (size_t)m * e.ldo + n;
        e.resid[i] = load_fresh(e.resid, i) + v;
        return;
    }
    if (e.mode == EPI_QKV && n >= e.d_model) {
        int c = n - e.d_model;
        __half *cache = e.kc;
        if (c >= e.d_model) {
            c -= e.d_model;
            cache = e.vc;
        }
        int head = c >> 6, el = c & 63;
        int b = m / e.rows_per_seq, s = m - b * e.rows_per_seq;
        int pos = (e.pos_ptr ? load_fresh_int(e.pos_ptr) : 0) + e.pos_off + s;
        if (pos < e.cap) cache[(((size_t)b * e.n_head + head) * e.cap + pos) * 64 + el] = __float2half_rn(v);
        return;
    }
    v = apply_act(v, e.act);
    if (B16 && e.row_scale) v *= load_fresh(e.row_scale, (size_t)m * e.rs_ld + n / e.rs_cols);
    size_t i = (size_t)m * e.ldo + n;
    if (B16 && e.out_half == OUT_BF16)
        static_cast<__nv_bfloat16 *>(e.out)[i] = __float2bfloat16_rn(v);
    else if (e.out_half)
        static_cast<__half *>(e.out)[i] = __float2half_rn(v);
    else
        static_cast<float *>(e.out)[i] = v;
}

// U token rows' finished values at once, the activation chosen once for all of them.
template <int ACT, int U>
__device__ __forceinline__ void act_rows(float4 (&v)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
        v[u].x = apply_act(v[u].x, ACT); v[u].y = apply_act(v[u].y, ACT);
        v[u].z = apply_act(v[u].z, ACT); v[u].w = apply_act(v[u].w, ACT);
    }
}
template <int U>
__device__ __forceinline__ void act_rows(float4 (&v)[U], int act) {
    switch (act) {
        case B200NN_ACT_GELU_TANH: return act_rows<B200NN_ACT_GELU_TANH>(v);
        case B200NN_ACT_GELU_SIGMOID: return act_rows<B200NN_ACT_GELU_SIGMOID>(v);
        case B200NN_ACT_RELU: return act_rows<B200NN_ACT_RELU>(v);
        case B200NN_ACT_SILU: return act_rows<B200NN_ACT_SILU>(v);
        case B200NN_ACT_SIGMOID: return act_rows<B200NN_ACT_SIGMOID>(v);
        default: return;
    }
}

// Four consecutive columns n..n+3 (n % 4 == 0) of the token rows m0, m0 + step, ... (cnt <= U of them; values past cnt are
// not looked at): 16-byte (f32) or 8-byte (fp16) stores when the destination allows it, element-wise otherwise.  pos_ptr
// must already be folded into e.pos_off by the caller (it is not dereferenced here for the vector path).
// What to do with a value is decided once for the U rows, and their chains (activation, position, rotation) run under each
// other (the hybrid decoder's prompts of 64 x 1024 and 32 steps: 50.2 -> 49.1 ms with four rows).
template <int U, bool B16 = false>
__device__ __forceinline__ void epi_store4_rows(const Epilogue &e, int m0, int step, int cnt, int n, float4 (&v)[U], int N) {
    if (e.no_store) return;
    if (B16 && e.mode == EPI_GLU) { // N and ldo are multiples of 4
        if (n >= N) return;
        float4 g[U];
#pragma unroll
        for (int u = 0; u < U; ++u) g[u] = make_float4(v[u].x, v[u].y, 0.0f, 0.0f);
        act_rows<U>(g, e.act);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < cnt)
                *reinterpret_cast<uint32_t *>(static_cast<__nv_bfloat16 *>(e.out) + (size_t)(m0 + u * step) * e.ldo + (n >> 1)) =
                    pack_bf16x2(g[u].x * v[u].z, g[u].y * v[u].w);
        return;
    }
    if (B16 && e.mode == EPI_ROPE) {
        if (n >= N) return;
        const int p = (n % e.rope_head - e.rope_at) >> 1;
        if (p >= 0 && p < e.rope_pairs) {
            float2 c0[U], c1[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float2 *t = e.rope_tab + (size_t)row_pos(e.rows, m0 + (u < cnt ? u : 0) * step) * e.rope_pairs + p;
                c0[u] = t[0];
                c1[u] = p + 1 < e.rope_pairs ? t[1] : make_float2(1.0f, 0.0f);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                v[u] = make_float4(v[u].x * c0[u].x - v[u].y * c0[u].y, v[u].y * c0[u].x + v[u].x * c0[u].y,
                                   v[u].z * c1[u].x - v[u].w * c1[u].y, v[u].w * c1[u].x + v[u].z * c1[u].y);
        }
    }
    if (B16 && e.tail_out && n >= e.tail_at) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u >= cnt) break;
            const float f[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
            const size_t i = (size_t)(m0 + u * step) * e.tail_ld + (n - e.tail_at);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < N) {
                    if (e.tail_type == OUT_BF16) static_cast<__nv_bfloat16 *>(e.tail_out)[i + j] = __float2bfloat16_rn(f[j]);
                    else static_cast<float *>(e.tail_out)[i + j] = f[j];
                }
        }
        return;
    }
    if (B16 && e.kv_cache && n >= e.kv_at) { // kv_w is a multiple of 16
        if (n >= N) return;
        const int c = n - e.kv_at, head = c / e.kv_w;
        int pos[U], slot[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int m = m0 + (u < cnt ? u : 0) * step;
            pos[u] = row_pos(e.rows, m);
            slot[u] = row_slot(e.rows, m);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < cnt) {
                const size_t row = ((size_t)slot[u] * e.kv_heads + head) * e.kv_cap + pos[u];
                *reinterpret_cast<uint2 *>(e.kv_cache + row * e.kv_w + (c - head * e.kv_w)) =
                    make_uint2(pack_bf16x2(v[u].x, v[u].y), pack_bf16x2(v[u].z, v[u].w));
            }
        return;
    }
    const bool vec = (n + 3 < N) && ((e.ldo & 3) == 0) && (e.pos_ptr == nullptr);
    if (!vec) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u >= cnt) break;
            if (n < N) epi_store<B16>(e, m0 + u * step, n, v[u].x);
            if (n + 1 < N) epi_store<B16>(e, m0 + u * step, n + 1, v[u].y);
            if (n + 2 < N) epi_store<B16>(e, m0 + u * step, n + 2, v[u].z);
            if (n + 3 < N) epi_store<B16>(e, m0 + u * step, n + 3, v[u].w);
        }
        return;
    }
    if (e.mode == EPI_RESID) {
        float4 r[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < cnt) r[u] = load_fresh4(e.resid + (size_t)(m0 + u * step) * e.ldo + n);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < cnt) *reinterpret_cast<float4 *>(e.resid + (size_t)(m0 + u * step) * e.ldo + n) = f4_add(r[u], v[u]);
        return;
    }
    if (e.mode == EPI_QKV && n >= e.d_model) {
        int c = n - e.d_model;
        __half *cache = e.kc;
        if (c >= e.d_model) {
            c -= e.d_model;
            cache = e.vc;
        }
        cache += (size_t)(c >> 6) * e.cap * 64 + (c & 63);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int m = m0 + u * step, b = e.rows_per_seq == 1 ? m : m / e.rows_per_seq, pos = e.pos_off + m - b * e.rows_per_seq;
            if (u < cnt && pos < e.cap)
                *reinterpret_cast<uint2 *>(cache + ((size_t)b * e.n_head * e.cap + pos) * 64) =
                    make_uint2(pack_f16x2(v[u].x, v[u].y), pack_f16x2(v[u].z, v[u].w));
        }
        return;
    }
    act_rows<U>(v, e.act);
    if (B16 && e.row_scale) {
        float rs[U];
#pragma unroll
        for (int u = 0; u < U; ++u) rs[u] = load_fresh(e.row_scale, (size_t)(m0 + (u < cnt ? u : 0) * step) * e.rs_ld + n / e.rs_cols);
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = make_float4(v[u].x * rs[u], v[u].y * rs[u], v[u].z * rs[u], v[u].w * rs[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (u >= cnt) break;
        const size_t i = (size_t)(m0 + u * step) * e.ldo + n;
        if (e.out_half) {
            *reinterpret_cast<uint2 *>(static_cast<__half *>(e.out) + i) =
                B16 && e.out_half == OUT_BF16 ? make_uint2(pack_bf16x2(v[u].x, v[u].y), pack_bf16x2(v[u].z, v[u].w))
                                              : make_uint2(pack_f16x2(v[u].x, v[u].y), pack_f16x2(v[u].z, v[u].w));
        } else {
            *reinterpret_cast<float4 *>(static_cast<float *>(e.out) + i) = v[u];
        }
    }
}

// ---- plain epilogues --------------------------------------------------------------------------------
// The epilogues that most tensor-core GEMMs of a pass have, each in a kernel of its own.  A block runs its epilogue once, so
// what it costs is mostly the fetching of its instructions and the chain of one row's decisions: with all modes in
// one kernel a token row took 900 cycles.  They want rows that leave as 16- or 8-byte pieces (N and ldo multiples of 4).
enum EpiKind {
    EK_ANY,   // every mode and shape
    EK_STORE, // y = sums + bias
    EK_GELU,  // the same through tanh-GELU (f32 or fp16)
    EK_QKV,   // fp16 q and cache rows
    EK_RESID, // splits added into the residual stream
    EK_ROWS,  // y = sums + bias in f32, rows of any length, greedy pick or not: the output matrix (int4 GEMM)
    EK_GLU    // act(gate) * up in bfloat16 (bfloat16 GEMM)
};
inline int epi_kind(const Epilogue &e, int N, int splits, bool b16) {
    if (e.ln_stats || e.row_scale || e.tail_out || e.kv_cache) return EK_ANY;
    if (e.mode == EPI_RESID) return splits > 1 ? EK_RESID : EK_ANY;
    if (!b16 && e.mode == EPI_STORE && splits == 1 && e.act == B200NN_ACT_NONE && e.out_half == OUT_F32 && (e.amax_val || ((N | e.ldo) & 3)))
        return EK_ROWS;
    if (e.no_store || e.amax_val || ((N | e.ldo) & 3) || splits > 8) return EK_ANY;
    if (b16 && e.mode == EPI_GLU) return e.act == B200NN_ACT_SILU || e.act == B200NN_ACT_GELU_TANH ? EK_GLU : EK_ANY;
    if (!b16 && e.mode == EPI_QKV) return e.out_half == OUT_F16 && e.act == B200NN_ACT_NONE && e.d_model % 64 == 0 ? EK_QKV : EK_ANY;
    if (e.mode != EPI_STORE || (!b16 && e.out_half == OUT_BF16)) return EK_ANY;
    return e.act == B200NN_ACT_NONE ? EK_STORE : !b16 && e.act == B200NN_ACT_GELU_TANH ? EK_GELU : EK_ANY;
}
// The finished sums of token rows m0, m0 + step, ... (cnt <= U), features n .. n+3 of each, for EK_STORE, EK_GELU, EK_QKV
// and EK_GLU.
template <int EK, int U, bool B16 = false>
__device__ __forceinline__ void plain_rows(const Epilogue &e, int pos_off, int m0, int step, int cnt, int n, float4 (&v)[U], float4 b4, int N) {
    if (n >= N) return;
    if constexpr (EK == EK_QKV) {
        const int part = n / e.d_model, c = n - part * e.d_model;
        __half *cache = (part == 1 ? e.kc : e.vc) + (size_t)(c >> 6) * e.cap * 64 + (c & 63);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int m = m0 + u * step, b = e.rows_per_seq == 1 ? m : m / e.rows_per_seq, pos = pos_off + m - b * e.rows_per_seq;
            if (u >= cnt || (part && pos >= e.cap)) continue;
            __half *dst = part ? cache + ((size_t)b * e.n_head * e.cap + pos) * 64 : static_cast<__half *>(e.out) + (size_t)m * e.ldo + n;
            *reinterpret_cast<uint2 *>(dst) = make_uint2(pack_f16x2(v[u].x + b4.x, v[u].y + b4.y), pack_f16x2(v[u].z + b4.z, v[u].w + b4.w));
        }
    } else if constexpr (EK == EK_GLU) {
        float4 g[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v[u] = f4_add(v[u], b4);
            g[u] = make_float4(v[u].x, v[u].y, 0.0f, 0.0f);
        }
        if (e.act == B200NN_ACT_SILU) act_rows<B200NN_ACT_SILU>(g);
        else act_rows<B200NN_ACT_GELU_TANH>(g);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < cnt)
                *reinterpret_cast<uint32_t *>(static_cast<__nv_bfloat16 *>(e.out) + (size_t)(m0 + u * step) * e.ldo + (n >> 1)) =
                    pack_bf16x2(g[u].x * v[u].z, g[u].y * v[u].w);
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            v[u] = f4_add(v[u], b4);
            if constexpr (EK == EK_GELU) v[u] = make_float4(gelu_tanh_f(v[u].x), gelu_tanh_f(v[u].y), gelu_tanh_f(v[u].z), gelu_tanh_f(v[u].w));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u >= cnt) continue;
            const size_t i = (size_t)(m0 + u * step) * e.ldo + n;
            if (e.out_half)
                *reinterpret_cast<uint2 *>(static_cast<__half *>(e.out) + i) =
                    B16 && e.out_half == OUT_BF16 ? make_uint2(pack_bf16x2(v[u].x, v[u].y), pack_bf16x2(v[u].z, v[u].w))
                                                  : make_uint2(pack_f16x2(v[u].x, v[u].y), pack_f16x2(v[u].z, v[u].w));
            else
                *reinterpret_cast<float4 *>(static_cast<float *>(e.out) + i) = v[u];
        }
    }
}

// ---- greedy pick fused into the epilogue ---------------------------------------------------------
// The better of two (value, index) candidates: larger value; on equal values the lower index, or the
// higher with keep_last (Rust's max_by, gpt2.rs:991-997).  NaN never wins, as in argmax_kernel.
__device__ __forceinline__ void amax_merge(float &bv, int &bi, float v, int i, int keep_last) {
    if (v > bv || (v == bv && (keep_last ? i > bi : i < bi))) {
        bv = v;
        bi = i;
    }
}
// Warp-collective (all 32 lanes, converged).  The lane holds the finished values of features n..n+3 of
// row m (n a multiple of 4, consecutive lanes consecutive groups of four): each group of eight lanes
// covers 32 features = one entry of the partial-argmax table.
__device__ __forceinline__ void epi_argmax4(const Epilogue &e, int m, int n, float4 v, int N) {
    float bv = -INFINITY;
    int bi = e.amax_keep_last ? -1 : 0x7fffffff;
    if (n < N) amax_merge(bv, bi, v.x, n, e.amax_keep_last);
    if (n + 1 < N) amax_merge(bv, bi, v.y, n + 1, e.amax_keep_last);
    if (n + 2 < N) amax_merge(bv, bi, v.z, n + 2, e.amax_keep_last);
    if (n + 3 < N) amax_merge(bv, bi, v.w, n + 3, e.amax_keep_last);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        amax_merge(bv, bi, ov, oi, e.amax_keep_last);
    }
    if ((threadIdx.x & 7) == 0 && (n >> 5) < e.amax_entries) {
        const size_t at = (size_t)m * e.amax_entries + (n >> 5);
        e.amax_val[at] = bv;
        e.amax_idx[at] = bi;
    }
}
// Warp-collective.  The lane holds the finished value of feature n of row m, the warp 32 consecutive
// features starting at a multiple of 32 (valid = the lane's feature exists).
__device__ __forceinline__ void epi_argmax1(const Epilogue &e, int m, int n, float v, bool valid) {
    float bv = valid ? v : -INFINITY;
    int bi = valid && v == v ? n : (e.amax_keep_last ? -1 : 0x7fffffff);
    if (!(bv == bv)) bv = -INFINITY; // NaN never wins
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        amax_merge(bv, bi, ov, oi, e.amax_keep_last);
    }
    if ((threadIdx.x & 31) == 0 && (n >> 5) < e.amax_entries) {
        const size_t at = (size_t)m * e.amax_entries + (n >> 5);
        e.amax_val[at] = bv;
        e.amax_idx[at] = bi;
    }
}

// Bias of the four features n..n+3 (zero without a bias and past N).
__device__ __forceinline__ float4 epi_bias4(const Epilogue &e, int n, int N) {
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (e.bias) {
        if (n < N) b.x = e.bias[n];
        if (n + 1 < N) b.y = e.bias[n + 1];
        if (n + 2 < N) b.z = e.bias[n + 2];
        if (n + 3 < N) b.w = e.bias[n + 3];
    }
    return b;
}

// Residual epilogue as a reduction at L2: resid[m, n..n+3] += v with one vector `red` (no load for
// the warp to wait on), element-wise atomics where the row is not 16-byte aligned or crosses N.
// Several K splits may add to the same element; the order of their additions is then not fixed.
__device__ __forceinline__ void epi_resid_red4(const Epilogue &e, int m, int n, float4 v, int N) {
    float *dst = e.resid + (size_t)m * e.ldo + n;
    if ((n + 3 < N) && ((e.ldo & 3) == 0)) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                     : "memory");
    } else {
        if (n < N) atomicAdd(dst, v.x);
        if (n + 1 < N) atomicAdd(dst + 1, v.y);
        if (n + 2 < N) atomicAdd(dst + 2, v.z);
        if (n + 3 < N) atomicAdd(dst + 3, v.w);
    }
}

// ---- LayerNorm folded into the neighbouring GEMMs (see Epilogue) ---------------------------------
// A row's (mean, 1/sqrt(var + eps)) from the partial sums its producer left, added in tile order.
__device__ __forceinline__ float2 epi_row_mean_rstd(const Epilogue &e, int m) {
    const float2 *p = reinterpret_cast<const float2 *>(e.ln_stats) + (size_t)m * e.ln_nt;
    float s1 = 0.0f, s2 = 0.0f;
    for (int j = 0; j < e.ln_nt; ++j) {
        const float2 v = __ldcg(p + j);
        s1 += v.x;
        s2 += v.y;
    }
    const float mean = s1 * e.ln_inv_d;
    return make_float2(mean, rsqrtf(fmaxf(s2 * e.ln_inv_d - mean * mean, 0.0f) + e.ln_eps));
}
// The four sums of products acc (features n..n+3 of a row) -> finished values: plain bias add, or with
// ln_stats the normalisation applied after the product (mr = the row's mean and rstd, g4 =
// ln_gsum[n..n+3], b4 = bias[n..n+3]).
__device__ __forceinline__ float4 epi_finish4(const Epilogue &e, float4 acc, float4 g4, float4 b4, float2 mr) {
    if (!e.ln_stats) return f4_add(acc, b4);
    const float mean = mr.x, rstd = mr.y;
    return make_float4(fmaf(rstd, fmaf(-mean, g4.x, acc.x), b4.x), fmaf(rstd, fmaf(-mean, g4.y, acc.y), b4.y),
                       fmaf(rstd, fmaf(-mean, g4.z, acc.z), b4.z), fmaf(rstd, fmaf(-mean, g4.w, acc.w), b4.w));
}
// The per-lane constant of the LayerNorm fold: the consumer's ln_gsum[n..n+3], or the producer's
// next_g[n..n+3] (no Linear is both).
__device__ __forceinline__ float4 epi_fold4(const Epilogue &e, int n, int N) {
    const float *src = e.mode == EPI_RESID_LN ? e.next_g : e.ln_gsum;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (src) {
        if (n < N) g.x = src[n];
        if (n + 1 < N) g.y = src[n + 1];
        if (n + 2 < N) g.z = src[n + 2];
        if (n + 3 < N) g.w = src[n + 3];
    }
    return g;
}
// The residual values a producer row will be added to (fetched early, under the reduction of the sums).
__device__ __forceinline__ float4 epi_resid_old4(const Epilogue &e, int m, int n, int N) {
    if (e.mode != EPI_RESID_LN || n >= N) return make_float4(0.f, 0.f, 0.f, 0.f);
    return load_fresh4(e.resid + (size_t)m * e.ldo + n);
}
// Residual epilogue that also prepares the next LayerNorm.  Warp-collective: the 32 lanes are converged on
// one token row m, lane l holding features n..n+3 (n = 128 * tile + 4 l); v = the finished values (bias
// included), r = epi_resid_old4, ng = next_g[n..n+3].  N and ldo are multiples of 4 (the model width).
__device__ __forceinline__ void epi_resid_ln4(const Epilogue &e, int m, int n, float4 v, float4 r, float4 ng, int N) {
    float s1 = 0.0f, s2 = 0.0f;
    if (n < N) {
        const size_t i = (size_t)m * e.ldo + n;
        r.x += v.x; r.y += v.y; r.z += v.z; r.w += v.w;
        *reinterpret_cast<float4 *>(e.resid + i) = r;
        __half2 lo = __floats2half2_rn(r.x * ng.x, r.y * ng.y), hi = __floats2half2_rn(r.z * ng.z, r.w * ng.w);
        *reinterpret_cast<uint2 *>(e.xg_out + i) = make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
        s1 = (r.x + r.y) + (r.z + r.w);
        s2 = (r.x * r.x + r.y * r.y) + (r.z * r.z + r.w * r.w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if ((threadIdx.x & 31) == 0)
        *reinterpret_cast<float2 *>(e.stats_out + ((size_t)m * e.stats_nt + (n >> 7)) * 2) = make_float2(s1, s2);
}
// cnt <= U finished rows (m0, m0 + step, ...) of a 128-feature tile leave the GEMM (warp-collective): v = the complete sums,
// bias not yet added.
template <int U, bool B16 = false>
__device__ __forceinline__ void epi_emit4_rows(const Epilogue &e2, const Epilogue &epi, int m0, int step, int cnt, int n, float4 (&v)[U],
                                               float4 b4, int N) {
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = f4_add(v[u], b4);
    if (epi.amax_val)
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < cnt) epi_argmax4(epi, m0 + u * step, n, v[u], N);
    epi_store4_rows<U, B16>(e2, m0, step, cnt, n, v, N);
}
// One finished row of a 128-feature tile leaves the GEMM (warp-collective as above): acc = the complete
// sums of products, f4 = epi_fold4, mr = the row's (mean, rstd) when ln_stats is set, r = epi_resid_old4.
__device__ __forceinline__ void epi_emit4(const Epilogue &e2, const Epilogue &epi, int m, int n, float4 acc, float4 f4,
                                          float4 b4, float2 mr, float4 r, int N) {
    float4 v[1] = {epi_finish4(epi, acc, f4, b4, mr)};
    if (epi.mode == EPI_RESID_LN) {
        epi_resid_ln4(epi, m, n, v[0], r, f4, N);
    } else {
        epi_store4_rows<1>(e2, m, 1, 1, n, v, N);
        v[0] = epi_finish4(epi, acc, f4, b4, mr);
        if (epi.amax_val) epi_argmax4(epi, m, n, v[0], N);
    }
}

// Same, from a raw accumulated dot product.
template <bool B16 = false>
__device__ __forceinline__ void epi_apply(const Epilogue &e, int m, int n, float acc) {
    epi_store<B16>(e, m, n, acc + (e.bias ? e.bias[n] : 0.0f));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over the block; every thread gets the result.  red must hold 32 floats.
__device__ __forceinline__ float block_sum(float v, float *red) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    float t = (lane < nw) ? red[lane] : 0.0f;
    return warp_sum(t);
}

template <typename T>
__device__ __forceinline__ float load_as_float(const T *p, size_t i);
template <>
__device__ __forceinline__ float load_as_float<float>(const float *p, size_t i) { return p[i]; }
template <>
__device__ __forceinline__ float load_as_float<__half>(const __half *p, size_t i) { return __half2float(p[i]); }
template <>
__device__ __forceinline__ float load_as_float<__nv_bfloat16>(const __nv_bfloat16 *p, size_t i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void store_from_float(float *p, float v) { *p = v; }
__device__ __forceinline__ void store_from_float(__half *p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void store_from_float(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

// The two halves of a cluster-wide barrier, and a store into the same shared variable of another block of the cluster.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster(float *p, int rank, float v) {
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.f32 [a], %2;\n\t}" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(p)),
                 "r"(rank), "f"(v)
                 : "memory");
}

// LayerNorm of up to MT f32 rows x [m_valid][K] (K <= NORM_IN_MAX) by one block: the values of columns k0 .. k0+cols go
// to xs [MT][ld] (zero past them and past m_valid).  Mean, then the mean square about it, as layernorm_kernel has it.
// Contains the wait on the previous kernel, after the loads of scale and shift.  red: THREADS / 32 * MT floats; the
// caller synchronises before it reads xs or reuses red.
// held: null, or [MT + 2][K] floats of shared memory in which the threads keep their values, scale and shift between the
// sums, for kernels whose registers are full of weights (each thread reads back what it wrote itself).
template <int MT, int THREADS, bool HELD = false>
__device__ __forceinline__ void norm_rows_to_smem(const NormIn &ln, Fresh<float> x, int m_valid, int K, int k0, int cols,
                                                  int ld, float *xs, float *red, float *held = nullptr) {
    constexpr int VPT = NORM_IN_MAX / THREADS, WARPS = THREADS / 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float regs[HELD ? 1 : MT + 2][HELD ? 1 : VPT], s[MT];
    auto put = [&](int row, int i, float v) {
        if constexpr (HELD) {
            if (tid + i * THREADS < K) held[row * K + tid + i * THREADS] = v;
        } else {
            regs[row][i] = v;
        }
    };
    auto get = [&](int row, int i) { // 0 past K
        if constexpr (HELD) return tid + i * THREADS < K ? held[row * K + tid + i * THREADS] : 0.0f;
        else return regs[row][i];
    };
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int k = tid + i * THREADS;
        const bool mine = k >= k0 && k < k0 + cols;
        put(MT, i, mine ? __ldg(ln.g + k) : 0.0f);
        put(MT + 1, i, mine ? __ldg(ln.b + k) : 0.0f);
    }
    pdl_wait();
    auto sums = [&]() { // s[m] over the block, divided by K
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            s[m] = warp_sum(s[m]);
            if (lane == 0) red[warp * MT + m] = s[m];
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            float t = 0.0f;
#pragma unroll
            for (int wi = 0; wi < WARPS; ++wi) t += red[wi * MT + m];
            s[m] = t / (float)K;
        }
        __syncthreads();
    };
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        s[m] = 0.0f;
        float v[VPT];
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int k = tid + i * THREADS;
            v[i] = m < m_valid && k < K ? x[(size_t)m * K + k] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            put(m, i, v[i]);
            s[m] += v[i];
        }
    }
    sums();
    float mean[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        mean[m] = s[m];
        s[m] = 0.0f;
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const float t = tid + i * THREADS < K ? get(m, i) - mean[m] : 0.0f;
            s[m] += t * t;
        }
    }
    sums();
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const float inv_std = rsqrtf(s[m] + ln.eps);
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            const int kk = tid + i * THREADS - k0;
            if (kk >= 0 && kk < ld) xs[m * ld + kk] = m < m_valid && kk < cols ? (get(m, i) - mean[m]) * inv_std * get(MT, i) + get(MT + 1, i) : 0.0f;
        }
    }
}

// Columns k0 .. k0+cols of up to MT rows x [m_valid][K] as f32 in xs [MT][ld], zero past them and past m_valid.  The rows
// are requested together (one after the other, each waited out its own latency: four rows, int4 768 x 2304 4.0 -> 3.3 us,
// f32 3072 x 768 20.5 -> 18.3).
template <int MT, int THREADS, typename XT>
__device__ __forceinline__ void rows_to_smem(Fresh<XT> x, int m_valid, int K, int k0, int cols, int ld, float *xs) {
    constexpr int U = MT == 4 ? 2 : 4; // columns of a thread in flight, MT loads each
    for (int base = threadIdx.x; base < ld; base += U * THREADS) {
        float v[U][MT];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int m = 0; m < MT; ++m)
                v[u][m] = m < m_valid && base + u * THREADS < cols ? x[(size_t)m * K + k0 + base + u * THREADS] : 0.0f;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int m = 0; m < MT; ++m)
                if (base + u * THREADS < ld) xs[m * ld + base + u * THREADS] = v[u][m];
    }
}

__device__ __forceinline__ float sigmoid_f(float v) { return 1.0f / (1.0f + expf(-v)); }

// Pairs of f32 in one register pair: one instruction for two multiply-adds.
__device__ __forceinline__ uint64_t f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f32x2_parts(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

// Unpacks one 32-bit word of the tiled int4 layout (nibble positions 0..7 = k offsets
// 0,2,4,6,1,3,5,7, each stored +8) into four half2 holding the exact integers (k0,k1) (k2,k3)
// (k4,k5) (k6,k7) in [-8,7].
__device__ __forceinline__ void unpack8_int4(uint32_t w, __half2 (&q)[4]) {
    const uint32_t MAGIC = 0x64006400u; // 1024.0 in both halves
    uint32_t h0, h1, h2, h3;
    asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xea;" : "=r"(h0) : "r"(w), "r"(MAGIC));
    asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xea;" : "=r"(h1) : "r"(w), "r"(MAGIC));
    uint32_t w8 = w >> 8;
    asm("lop3.b32 %0, %1, 0x000f000f, %2, 0xea;" : "=r"(h2) : "r"(w8), "r"(MAGIC));
    asm("lop3.b32 %0, %1, 0x00f000f0, %2, 0xea;" : "=r"(h3) : "r"(w8), "r"(MAGIC));
    const __half2 c1032 = __floats2half2_rn(1032.0f, 1032.0f);
    const __half2 c16th = __floats2half2_rn(0.0625f, 0.0625f);
    const __half2 cm72 = __floats2half2_rn(-72.0f, -72.0f);
    q[0] = __hsub2(*reinterpret_cast<__half2 *>(&h0), c1032);       // (1024+n) - 1032
    q[1] = __hfma2(*reinterpret_cast<__half2 *>(&h1), c16th, cm72); // (1024+16n)/16 - 72
    q[2] = __hsub2(*reinterpret_cast<__half2 *>(&h2), c1032);
    q[3] = __hfma2(*reinterpret_cast<__half2 *>(&h3), c16th, cm72);
}
