// Gated delta rule: a linear-attention recurrence whose state is one [dim, vdim] f32 matrix per head and
// sequence.  Per token S <- g S, u = beta (v - S^T k), S <- S + k u^T, o = S^T q.  Both products against S are
// taken on the state before the write: S_new^T q = g S^T q + (k . q) u, so a token costs one pass over the
// state and one reduction instead of two.  Everything here is f32.
//
// The decay g is one number per head, or (CH, DeltaDims::channel) one per head and key channel, acting on the rows of
// S; the output gate is then a sigmoid and its input, like the decays', comes from a projection of its own (`ext`).
//
//   delta_step_kernel     decoding: convolution, norms, recurrence, output norm and gate of one token
//   delta_conv_kernel     prompts: convolution + silu, unit norms, k . q, decay and step size of every row
//   delta_scan_kernel     prompts: the recurrence (state columns are independent: a block owns some of them)
//   delta_out_kernel      prompts: output norm and gate
//
// The convolution's inputs are kept in a ring of `taps` rows per slot (position p in row p % taps): a token
// reads the other rows and replaces its own, so heads that share a query/key head do not race.
#include <algorithm>

#include <cuda.h>

#include "device_utils.cuh"
#include "hybrid.h"
#include "tc_ptx.cuh"

namespace {

// activation of the convolution and of the output gate (not part of the recurrence): fast exponential and division
__device__ __forceinline__ float silu_f(float v) { return __fdividef(v, 1.0f + __expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.0f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float decay_f(float a_exp, float a, float dt_bias) { return expf(-a_exp * softplus_f(a + dt_bias)); }

// ---- decoding ----------------------------------------------------------------------------------------
// Block = (row, head), eight warps.  Warp w holds state rows w, w + 8, ...; lane l columns 4l .. 4l+3 of a
// 128-column chunk (one chunk for vdim <= 128).  Under the state's loads warps 0, 1 and 2 make the query, key and value
// (a lane takes four channels; the unit norms stay scalar factors), warp 3 gate times norm weight, warp 4 decay and
// step size.
template <int RPW, bool CH, typename T>
__global__ void __launch_bounds__(256, RPW <= 16 ? 2 : 1)
delta_step_kernel(DeltaDims d, Fresh<float> proj, int ldp, Fresh<float> ext, DeltaWeights w, float *__restrict__ conv_state,
                  float *__restrict__ state, RowMap rows, T *__restrict__ out) {
    // q [dim_p], k [dim_p], v, gate, o [vdim_p], reduction [8][2][128], scalars [8], CH: decays [dim_p]
    extern __shared__ __align__(16) float sh[];
    const int h = blockIdx.x, row = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float *sq = sh, *sk = sq + d.dim_p, *sv = sk + d.dim_p, *sgn = sv + d.vdim_p, *so = sgn + d.vdim_p, *red = so + d.vdim_p, *sc = red + 2048;
    float *sg = sc + 8;
    pdl_trigger();
    // Where the slot is the row number, the state can start its way to L2 under the kernel before (only a hint: nothing is read
    // until that kernel has ended).  64 rows of 8 heads of 128: 21.0 -> 17.4 us (state read and written: 10.4).
    if (!rows.slot && tid == 0) tc::bulk_prefetch_l2(state + ((size_t)row * d.heads + h) * d.dim_p * d.vdim_p, d.dim_p * d.vdim_p * 4);
    pdl_wait();
    const int pos = row_pos(rows, row), slot = row_slot(rows, row);
    float *S = state + ((size_t)slot * d.heads + h) * d.dim_p * d.vdim_p;
    float4 st[RPW];
    auto load_chunk = [&](int c0) {
        const bool col = c0 + lane * 4 < d.vdim_p;
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const int i = warp + 8 * r;
            st[r] = col && i < d.dim_p && pos > 0 ? load_fresh4(S + (size_t)i * d.vdim_p + c0 + lane * 4)
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    load_chunk(0);

    const Fresh<float> p = proj + (size_t)row * ldp;
    const int group = d.heads / d.kv_heads, kh = h / group;
    const int cw = d.conv_w(), here = pos % d.taps;
    float *cring = conv_state + (size_t)slot * d.taps * cw;
    // four channels: the inputs of up to four taps are requested together, then summed; keep: put the input into the ring
    struct Taps {
        float4 x[4], w[4];
    };
    auto request = [&](int ch) {
        Taps t;
        t.x[0] = p.four(ch);
        t.w[0] = __ldg(reinterpret_cast<const float4 *>(w.conv + (size_t)(d.taps - 1) * cw + ch));
#pragma unroll
        for (int i = 1; i < 4; ++i) {
            const bool use = i < d.taps && pos >= i;
            const int at = use ? (here - i < 0 ? here - i + d.taps : here - i) : here, tap = use ? d.taps - 1 - i : d.taps - 1;
            const float4 y = load_fresh4(cring + (size_t)at * cw + ch);
            t.x[i] = use ? y : make_float4(0.f, 0.f, 0.f, 0.f);
            t.w[i] = __ldg(reinterpret_cast<const float4 *>(w.conv + (size_t)tap * cw + ch));
        }
        return t;
    };
    auto channels = [&](const Taps &t, int ch, bool keep) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a.x = fmaf(t.x[i].x, t.w[i].x, a.x); a.y = fmaf(t.x[i].y, t.w[i].y, a.y);
            a.z = fmaf(t.x[i].z, t.w[i].z, a.z); a.w = fmaf(t.x[i].w, t.w[i].w, a.w);
        }
        for (int i = 4; i < d.taps && pos >= i; ++i) {
            const float4 y = load_fresh4(cring + (size_t)(here - i < 0 ? here - i + d.taps : here - i) * cw + ch);
            const float4 wt = __ldg(reinterpret_cast<const float4 *>(w.conv + (size_t)(d.taps - 1 - i) * cw + ch));
            a.x = fmaf(y.x, wt.x, a.x); a.y = fmaf(y.y, wt.y, a.y); a.z = fmaf(y.z, wt.z, a.z); a.w = fmaf(y.w, wt.w, a.w);
        }
        if (keep) *reinterpret_cast<float4 *>(cring + (size_t)here * cw + ch) = t.x[0];
        return make_float4(silu_f(a.x), silu_f(a.y), silu_f(a.z), silu_f(a.w));
    };
    if (warp < 3) { // query, key, value
        const int n = warp < 2 ? d.dim_p : d.vdim_p, at = warp == 0 ? d.q_at() + kh * d.dim_p : warp == 1 ? d.k_at() + kh * d.dim_p : d.v_at() + h * d.vdim_p;
        float *dst = warp == 0 ? sq : warp == 1 ? sk : sv;
        float s = 0.0f;
        for (int j = lane * 4; j < n; j += 128) {
            const float4 a = channels(request(at + j), at + j, warp == 2 || h % group == 0);
            *reinterpret_cast<float4 *>(dst + j) = a;
            s += (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
        }
        s = warp_sum(s);
        if (lane == 0) sc[2 + warp] = 1.0f / sqrtf(s + 1e-6f); // unit norms (the value's is not used)
    } else if (warp == 3) {
        for (int j = lane * 4; j < d.vdim_p; j += 128) { // the last columns may be padding: no norm weight there
            const Fresh<float> gate = CH ? ext + ((size_t)row * 2 * d.ext() + d.ext()) : p + d.g_at();
            const float4 gg = gate.four(h * d.vdim_p + j);
            const float e[4] = {gg.x, gg.y, gg.z, gg.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) sgn[j + i] = j + i < d.vdim ? w.norm[j + i] * (CH ? sigmoid_f(e[i]) : silu_f(e[i])) : 0.0f;
        }
    } else if (CH && warp == 4) {
        if (lane == 0) sc[0] = sigmoid_f(p[d.b_at() + h]);
        const float a_exp = w.a_exp[h];
        for (int j = lane; j < d.dim_p; j += 32)
            sg[j] = decay_f(a_exp, ext[(size_t)row * 2 * d.ext() + h * d.dim_p + j], w.dt_bias[h * d.dim_p + j]);
    } else if (!CH && tid == 128) {
        sc[0] = sigmoid_f(p[d.b_at() + h]);
        sc[1] = decay_f(w.a_exp[h], p[d.a_at() + h], w.dt_bias[h]);
    }
    __syncthreads();
    const float beta = sc[0], g = CH ? 1.0f : sc[1], fq = sc[2] / sqrtf((float)d.dim), fk = sc[3]; // q also times dim^(-1/2)
    float kq = 0.0f; // warp 0, which makes the read-out, needs k . q
    if (warp == 0) {
        for (int j = lane; j < d.dim_p; j += 32) kq = fmaf(sk[j], sq[j], kq);
        kq = warp_sum(kq) * fq * fk;
    }
    for (int c0 = 0; c0 < d.vdim_p; c0 += 128) {
        if (c0) load_chunk(c0);
        float4 ak = make_float4(0.f, 0.f, 0.f, 0.f), aq = ak;
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const int i = warp + 8 * r;
            if (i < d.dim_p) {
                const float gi = CH ? sg[i] : 1.0f, k = CH ? gi * sk[i] : sk[i], q = CH ? gi * sq[i] : sq[i];
                ak.x = fmaf(st[r].x, k, ak.x); ak.y = fmaf(st[r].y, k, ak.y); ak.z = fmaf(st[r].z, k, ak.z); ak.w = fmaf(st[r].w, k, ak.w);
                aq.x = fmaf(st[r].x, q, aq.x); aq.y = fmaf(st[r].y, q, aq.y); aq.z = fmaf(st[r].z, q, aq.z); aq.w = fmaf(st[r].w, q, aq.w);
            }
        }
        *reinterpret_cast<float4 *>(red + (warp * 2) * 128 + lane * 4) = ak;
        *reinterpret_cast<float4 *>(red + (warp * 2 + 1) * 128 + lane * 4) = aq;
        __syncthreads();
        float4 tk = make_float4(0.f, 0.f, 0.f, 0.f), tq = tk;
#pragma unroll
        for (int i = 0; i < 8; ++i) tk = f4_add(tk, *reinterpret_cast<const float4 *>(red + (i * 2) * 128 + lane * 4));
        if (warp == 0)
#pragma unroll
            for (int i = 0; i < 8; ++i) tq = f4_add(tq, *reinterpret_cast<const float4 *>(red + (i * 2 + 1) * 128 + lane * 4));
        const int c = c0 + lane * 4;
        if (c < d.vdim_p) {
            const float4 v = *reinterpret_cast<const float4 *>(sv + c);
            const float gk = g * fk, gq = g * fq;
            const float4 u = make_float4(beta * (v.x - gk * tk.x), beta * (v.y - gk * tk.y), beta * (v.z - gk * tk.z), beta * (v.w - gk * tk.w));
#pragma unroll
            for (int r = 0; r < RPW; ++r) {
                const int i = warp + 8 * r;
                if (i < d.dim_p) {
                    const float k = sk[i] * fk, gi = CH ? sg[i] : g;
                    *reinterpret_cast<float4 *>(S + (size_t)i * d.vdim_p + c) =
                        make_float4(fmaf(k, u.x, gi * st[r].x), fmaf(k, u.y, gi * st[r].y), fmaf(k, u.z, gi * st[r].z), fmaf(k, u.w, gi * st[r].w));
                }
            }
            if (warp == 0)
                *reinterpret_cast<float4 *>(so + c) =
                    make_float4(fmaf(kq, u.x, gq * tq.x), fmaf(kq, u.y, gq * tq.y), fmaf(kq, u.z, gq * tq.z), fmaf(kq, u.w, gq * tq.w));
        }
        if (c0 + 128 < d.vdim_p) __syncthreads(); // red is used again
    }
    if (warp) return; // the read-out is warp 0's own
    __syncwarp();
    float s = 0.0f;
    for (int j = lane; j < d.vdim; j += 32) s = fmaf(so[j], so[j], s);
    const float rn = 1.0f / sqrtf(warp_sum(s) / (float)d.vdim + d.eps);
    for (int j = lane; j < d.vdim; j += 32) store_from_float(out + ((size_t)row * d.heads + h) * d.vdim_p + j, so[j] * rn * sgn[j]);
}

// ---- prompts -----------------------------------------------------------------------------------------
// Columns of the convolved rows: q (scaled), k, v as in the projection, then per head the decay and the step size,
// then per query/key head k . q; rows DeltaDims::conv_ld() apart.
//
// A warp takes four rows of one unit: a query/key head (both of its vectors) or a value head.  The eight warps of a
// block take neighbouring rows, which share their convolution inputs in L1 (hence an ordered launch).
// NCH: 128-channel chunks of a query/key head.
constexpr int CONV_ROWS = 4;
template <int NCH, bool CH>
__global__ void __launch_bounds__(256)
delta_conv_kernel(DeltaDims d, const float *__restrict__ proj, int ldp, const float *__restrict__ ext, DeltaWeights w, const float *__restrict__ conv_state, RowMap rows,
                  SeqMap sm, const int *__restrict__ row_seq, int n_rows, float *__restrict__ conv) {
    pdl_trigger();
    const int r_first = (blockIdx.y * 8 + (threadIdx.x >> 5)) * CONV_ROWS, u = blockIdx.x, lane = threadIdx.x & 31;
    const int cw = d.conv_w(), ld = d.conv_ld();
    int pos[CONV_ROWS], back[CONV_ROWS]; // position; rows of the same sequence before it in the pass
    const float *cring[CONV_ROWS];
#pragma unroll
    for (int r = 0; r < CONV_ROWS; ++r) {
        const int row = min(r_first + r, n_rows - 1);
        pos[r] = row_pos(rows, row);
        back[r] = row - sm.row0[row_seq[row]];
        cring[r] = conv_state + (size_t)row_slot(rows, row) * d.taps * cw;
    }
    // channels ch .. ch+3 of row r_first + r after convolution and silu
    auto channels = [&](int r, int ch) {
        const float *p = proj + (size_t)min(r_first + r, n_rows - 1) * ldp;
        const float4 x = *reinterpret_cast<const float4 *>(p + ch), w0 = __ldg(reinterpret_cast<const float4 *>(w.conv + (size_t)(d.taps - 1) * cw + ch));
        float4 a = make_float4(x.x * w0.x, x.y * w0.y, x.z * w0.z, x.w * w0.w);
        for (int t = 1; t < d.taps && pos[r] - t >= 0; ++t) {
            const float4 y = *reinterpret_cast<const float4 *>(back[r] >= t ? p - (size_t)t * ldp + ch : cring[r] + (size_t)((pos[r] - t) % d.taps) * cw + ch);
            const float4 wt = __ldg(reinterpret_cast<const float4 *>(w.conv + (size_t)(d.taps - 1 - t) * cw + ch));
            a.x = fmaf(y.x, wt.x, a.x); a.y = fmaf(y.y, wt.y, a.y); a.z = fmaf(y.z, wt.z, a.z); a.w = fmaf(y.w, wt.w, a.w);
        }
        return make_float4(silu_f(a.x), silu_f(a.y), silu_f(a.z), silu_f(a.w));
    };
    // the same for all four rows; four neighbours of one sequence with their inputs in the pass share seven loads
    const bool shared = d.taps <= 4 && back[0] >= 3 && back[CONV_ROWS - 1] == back[0] + CONV_ROWS - 1 && r_first + CONV_ROWS <= n_rows;
    auto rows4 = [&](int ch, float4 (&o)[CONV_ROWS]) {
        if (!shared) {
#pragma unroll
            for (int r = 0; r < CONV_ROWS; ++r) o[r] = channels(r, ch);
            return;
        }
        float4 x[CONV_ROWS + 3], wt[4];
#pragma unroll
        for (int i = 0; i < CONV_ROWS + 3; ++i) x[i] = *reinterpret_cast<const float4 *>(proj + (size_t)(r_first + i - 3) * ldp + ch);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            wt[t] = t < d.taps ? __ldg(reinterpret_cast<const float4 *>(w.conv + (size_t)(d.taps - 1 - t) * cw + ch)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < CONV_ROWS; ++r) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float4 y = x[3 + r - t];
                a.x = fmaf(y.x, wt[t].x, a.x); a.y = fmaf(y.y, wt[t].y, a.y); a.z = fmaf(y.z, wt[t].z, a.z); a.w = fmaf(y.w, wt[t].w, a.w);
            }
            o[r] = make_float4(silu_f(a.x), silu_f(a.y), silu_f(a.z), silu_f(a.w));
        }
    };
    if (u >= d.kv_heads) { // a value head
        const int h = u - d.kv_heads;
        for (int j = lane * 4; j < d.vdim_p; j += 128) {
            float4 v[CONV_ROWS];
            rows4(d.v_at() + h * d.vdim_p + j, v);
#pragma unroll
            for (int r = 0; r < CONV_ROWS; ++r)
                if (r_first + r < n_rows) *reinterpret_cast<float4 *>(conv + (size_t)(r_first + r) * ld + d.v_at() + h * d.vdim_p + j) = v[r];
        }
        if (lane < CONV_ROWS && r_first + lane < n_rows) {
            const float *p = proj + (size_t)(r_first + lane) * ldp;
            float *o = conv + (size_t)(r_first + lane) * ld;
            if (!CH) o[d.decay_at() + h] = decay_f(w.a_exp[h], p[d.a_at() + h], w.dt_bias[h]);
            o[d.beta_at() + h] = sigmoid_f(p[d.b_at() + h]);
        }
        if (CH) {
            const float a_exp = w.a_exp[h];
            for (int j = lane * 4; j < d.dim_p; j += 128) {
                const float4 b = __ldg(reinterpret_cast<const float4 *>(w.dt_bias + h * d.dim_p + j));
#pragma unroll
                for (int r = 0; r < CONV_ROWS; ++r) {
                    if (r_first + r >= n_rows) break;
                    const float4 a = *reinterpret_cast<const float4 *>(ext + (size_t)(r_first + r) * 2 * d.ext() + h * d.dim_p + j);
                    *reinterpret_cast<float4 *>(conv + (size_t)(r_first + r) * ld + d.decay_at() + h * d.dim_p + j) =
                        make_float4(decay_f(a_exp, a.x, b.x), decay_f(a_exp, a.y, b.y), decay_f(a_exp, a.z, b.z), decay_f(a_exp, a.w, b.w));
                }
            }
        }
        return;
    }
    const float q_scale = 1.0f / sqrtf((float)d.dim);
    float4 q[NCH][CONV_ROWS], k[NCH][CONV_ROWS];
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
        const int j = lane * 4 + 128 * c;
#pragma unroll
        for (int r = 0; r < CONV_ROWS; ++r) q[c][r] = k[c][r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j < d.dim_p) {
            rows4(d.q_at() + u * d.dim_p + j, q[c]);
            rows4(d.k_at() + u * d.dim_p + j, k[c]);
        }
    }
#pragma unroll
    for (int r = 0; r < CONV_ROWS; ++r) {
        float qq = 0.0f, kk = 0.0f, kq = 0.0f;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const float4 a = q[c][r], b = k[c][r];
            qq += (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
            kk += (b.x * b.x + b.y * b.y) + (b.z * b.z + b.w * b.w);
            kq += (a.x * b.x + a.y * b.y) + (a.z * b.z + a.w * b.w);
        }
        const float fq = q_scale / sqrtf(warp_sum(qq) + 1e-6f), fk = 1.0f / sqrtf(warp_sum(kk) + 1e-6f);
        const float dot = warp_sum(kq) * fq * fk;
        if (r_first + r >= n_rows) continue;
        float *o = conv + (size_t)(r_first + r) * ld;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const int j = lane * 4 + 128 * c;
            if (j < d.dim_p) {
                const float4 a = q[c][r], b = k[c][r];
                *reinterpret_cast<float4 *>(o + d.q_at() + u * d.dim_p + j) = make_float4(a.x * fq, a.y * fq, a.z * fq, a.w * fq);
                *reinterpret_cast<float4 *>(o + d.k_at() + u * d.dim_p + j) = make_float4(b.x * fk, b.y * fk, b.z * fk, b.w * fk);
            }
        }
        if (lane == 0) o[d.kq_at() + u] = dot;
    }
}

enum : uint32_t { ERR_SCAN = 0x401 };
constexpr int SCAN_TOKENS = 8, SCAN_THREADS = 8 * SCAN_TOKENS; // eight lanes make one of a stage's TOK / 2 x 2 cross products
template <int DM, int NC, bool CH>
struct alignas(128) ScanStage { // the parts that tensor copies fill start on 128 bytes
    static constexpr int TOK = SCAN_TOKENS, DP = DM * 32;
    float qk[TOK][2][DP], v[TOK][8 * NC], s[TOK][4], g[CH ? TOK : 1][CH ? DP : 4]; // s: decay, step size, k . q; g: decays
    float cross[TOK / 2][2]; // k1 . k2 and k1 . q2 of each pair
};

// Block = (8 NC state columns, head, sequence), two warps.  The eight lanes of a column group hold its dim entries
// 4 l + 32 m .. + 3 of NC columns each (f32 pairs along dim).  Tokens come through shared memory TOK at a time, the next
// TOK being copied under the current ones, and are taken in pairs: all four products (k, q of both tokens) are taken on
// the state before the pair,
//     u1 = beta1 (v1 - g1 S^T k1),               o1 = g1 S^T q1 + (k1 . q1) u1,
//     u2 = beta2 (v2 - g1 g2 S^T k2 - g2 (k1 . k2) u1),  o2 = g1 g2 S^T q2 + g2 (k1 . q2) u1 + (k2 . q2) u2,
//     S <- g1 g2 S + g2 k1 u1^T + k2 u2^T,
// one lane reduction for the eight values (transposing: each lane ends with one of them) and one chain for two tokens.
// The state is held divided by the decay G accumulated since it was last rescaled (S = G s), so that a token costs three
// multiply-adds per entry; a pair that brings G below 2^-20 applies its decays to the state instead.
// With CH the decays differ along dim and are multiplied in directly (one multiply more per entry); !PAIRS (CH only) takes its
// tokens one at a time.
// What bounds it: the packed multiply-adds read three different operand pairs and issue every 3 to 3.5 cycles (two when operands
// repeat): 96 of them and 60 other instructions per warp and pair; and, per stage, 600 cycles of copies announced, cross
// products and two barriers.  One token at a time, copies by cp.async, four warps a block: 16 sequences of 1024 tokens, 8 heads of
// 128, 591 us, now 515; one of 512 133 / 100; decays per channel 2 sequences of 250 67.6 / 61.5, 8 137 / 105, one
// at a time 32 287 / 289; up to 16 tokens of few sequences cost up to a microsecond more (2 of 16: 9.0 / 9.8).  Asking for the first stage ahead of
// the state's loads: 0.05 us less there, and 2 % more for 64 sequences of 100.  Tried: four lanes for two columns (half the reductions, half the warps: 506, and
// 170 for one sequence), plain multiply-adds (576), a bulk copy per token and vector (920: one lane issues them), the
// cross products with the pair (longer chains), pairs unrolled (spills).
// Also leaves the convolution's last inputs in the cache (blocks of column group 0).
template <int DM, int NC, bool CH, bool PAIRS>
__global__ void __launch_bounds__(SCAN_THREADS, DM > 4 ? 4 : 8)
delta_scan_kernel(const __grid_constant__ CUtensorMap map_qk, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_g,
                  DeltaDims d, const float *__restrict__ proj, int ldp, const float *__restrict__ conv, float *__restrict__ conv_state,
                  float *__restrict__ state, SeqMap sm, float *__restrict__ heads_out, uint32_t *__restrict__ dev_err) {
    static_assert(CH || PAIRS, "one decay a head: pairs are the faster way for any number of sequences");
    constexpr int TOK = SCAN_TOKENS, T = SCAN_THREADS, DP = DM * 32, CB = T / 8 * NC;
    using Stage = ScanStage<DM, NC, CH>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[2]; // a stage's copies have landed
    __shared__ int abort_flag;
    Stage *stages = reinterpret_cast<Stage *>(smem_raw + (-tc::smem_u32(smem_raw) & 127));
    pdl_trigger();
    const int cg = blockIdx.x, h = blockIdx.y, sidx = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int part = lane & 7, cl = (tid >> 3) * NC, col = cg * CB + cl; // NC columns from col on
    const int n = sm.n[sidx], past = sm.past[sidx], slot = sm.slot[sidx], row0 = sm.row0[sidx];
    const int group = d.heads / d.kv_heads, kh = h / group, cw = d.conv_w(), ldc = d.conv_ld();
    float *S = state + ((size_t)slot * d.heads + h) * d.dim_p * d.vdim_p + col;
    uint64_t s[NC][DM * 2];
#pragma unroll
    for (int m = 0; m < DM; ++m)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const int i = 32 * m + 4 * part + e;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const bool in = i < d.dim_p && past > 0 && col + c < d.vdim_p;
                s[c][2 * m + e / 2] = in ? f32x2(S[(size_t)i * d.vdim_p + c], S[(size_t)(i + 1) * d.vdim_p + c]) : 0ull;
            }
        }
    // the tokens' single values (the last warp): requested before a stage's work, put down after it
    const int one = (T / 32 - 1) * 32, st_t = (tid - one) >> 2, st_j = tid & 3;
    const bool fetches = tid >= one && st_j < 3 && !(CH && st_j == 0);
    const float *single = conv + (size_t)row0 * ldc + (st_j == 0 ? d.decay_at() + h : st_j == 1 ? d.beta_at() + h : d.kq_at() + kh);
    auto fetch = [&](int t0) { return fetches && t0 + st_t < n ? single[(size_t)(t0 + st_t) * ldc] : 0.0f; };
    // A box of TOK rows of each part (entries past dim arrive as zeros; rows past the sequence's last are not used).
    auto copy = [&](int t0, Stage &st, uint64_t *landed) {
        if (tid == 0) {
            const uint32_t bar = tc::smem_u32(landed);
            tc::mbar_expect_tx(bar, TOK * (DP * (CH ? 3 : 2) + CB) * 4);
            tc::tma_load_4d(tc::smem_u32(st.qk), &map_qk, 0, kh, 0, row0 + t0, bar);
            tc::tma_load_4d(tc::smem_u32(st.v), &map_v, cg * CB, h, 0, row0 + t0, bar);
            if constexpr (CH) tc::tma_load_4d(tc::smem_u32(st.g), &map_g, 0, h, 0, row0 + t0, bar);
        }
    };
    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < 2; ++i) tc::mbar_init(tc::smem_u32(&full[i]), 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    if (n > 0) copy(0, stages[0], &full[0]); // (a sequence of no rows waits for nothing)
    if (tid >= one) stages[0].s[st_t][st_j] = fetch(0);
    __syncthreads();
    float G = 1.0f;
    auto rescale = [&](float f) {
        const uint64_t f2 = f32x2(f, f);
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int m = 0; m < DM * 2; ++m) s[c][m] = mul2(f2, s[c][m]);
    };
    // what a lane ends with: S^T k1, q1, k2 or q2, of column `mine`
    const int type = part >> 1, mine = NC == 2 ? part & 1 : 0;
    const bool writer = (type & 1) && (NC == 2 || !(part & 1)) && col + mine < d.vdim_p;
    float *o = heads_out + ((size_t)(row0 + (type >> 1)) * d.heads + h) * d.vdim_p + col + mine;
    const size_t o_step = (size_t)d.heads * d.vdim_p;
    for (int t0 = 0, b = 0; t0 < n; t0 += TOK, b ^= 1) {
        if (t0 + TOK < n) copy(t0 + TOK, stages[b ^ 1], &full[b ^ 1]);
        const float next = fetch(t0 + TOK);
        Stage &st = stages[b];
        const int nt = min(TOK, n - t0);
        tc::mbar_wait(tc::smem_u32(&full[b]), t0 / (2 * TOK) & 1, &abort_flag, dev_err, ERR_SCAN);
        if (PAIRS && (nt & 1)) { // the last token's partner: nothing read, nothing written
            for (int j = tid; j < DP; j += T) {
                st.qk[nt][0][j] = st.qk[nt][1][j] = 0.0f;
                if constexpr (CH) st.g[nt][j] = 1.0f;
            }
            if (tid < CB) st.v[nt][tid] = 0.0f;
            if (tid < 3) st.s[nt][tid] = tid == 0 ? 1.0f : 0.0f;
            __syncthreads();
        }
        if constexpr (PAIRS) { // k1 . k2 (even groups) and k1 . q2 (odd ones) of pair `at`, k1 under the second token's decay
            const int g = tid >> 3, at = g & ~1;
            const float *y = st.qk[at + 1][~g & 1];
            uint64_t a[2] = {};
#pragma unroll
            for (int m = 0; m < DM; ++m) {
                ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&st.qk[at][1][32 * m + 4 * part]);
                const ulonglong2 z = *reinterpret_cast<const ulonglong2 *>(&y[32 * m + 4 * part]);
                if constexpr (CH) {
                    const ulonglong2 gg = *reinterpret_cast<const ulonglong2 *>(&st.g[at + 1][32 * m + 4 * part]);
                    x.x = mul2(x.x, gg.x);
                    x.y = mul2(x.y, gg.y);
                }
                a[0] = fma2(x.x, z.x, a[0]);
                a[1] = fma2(x.y, z.y, a[1]);
            }
            const float2 a0 = f32x2_parts(a[0]), a1 = f32x2_parts(a[1]);
            float dot = (a0.x + a0.y) + (a1.x + a1.y);
#pragma unroll
            for (int sh = 4; sh; sh >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, sh);
            if (part == 0) st.cross[at >> 1][g & 1] = dot;
            __syncthreads();
        }
        if constexpr (!PAIRS) {
#pragma unroll 2
            for (int t = 0; t < nt; ++t) {
                const float4 sc = *reinterpret_cast<const float4 *>(st.s[t]);
                uint64_t k[DM * 2];
                float r[2 * NC]; // s^T k of the NC columns, then s^T q
                {
                    uint64_t acc[2 * NC];
#pragma unroll
                    for (int i = 0; i < 2 * NC; ++i) acc[i] = 0ull;
#pragma unroll
                    for (int m = 0; m < DM; ++m) {
                        const int at = 32 * m + 4 * part;
                        const ulonglong2 gg = *reinterpret_cast<const ulonglong2 *>(&st.g[t][at]);
                        const ulonglong2 kk = *reinterpret_cast<const ulonglong2 *>(&st.qk[t][1][at]), qq = *reinterpret_cast<const ulonglong2 *>(&st.qk[t][0][at]);
                        k[2 * m] = kk.x;
                        k[2 * m + 1] = kk.y;
#pragma unroll
                        for (int e = 0; e < 2; ++e)
#pragma unroll
                            for (int c = 0; c < NC; ++c) {
                                s[c][2 * m + e] = mul2(e ? gg.y : gg.x, s[c][2 * m + e]);
                                acc[c] = fma2(s[c][2 * m + e], e ? kk.y : kk.x, acc[c]);
                                acc[NC + c] = fma2(s[c][2 * m + e], e ? qq.y : qq.x, acc[NC + c]);
                            }
                    }
#pragma unroll
                    for (int i = 0; i < 2 * NC; ++i) {
                        const float2 a = f32x2_parts(acc[i]);
                        r[i] = a.x + a.y;
                    }
                }
#pragma unroll
                for (int sh = 4, w = NC; sh; sh >>= 1, w >>= 1) {
                    const bool up = (lane & sh) != 0;
#pragma unroll
                    for (int i = 0; i < w; ++i) {
                        const float send = up ? r[i] : r[i + w], keep = up ? r[i + w] : r[i];
                        r[i] = keep + __shfl_xor_sync(0xffffffffu, send, sh);
                    }
                    if (w == 0) r[0] += __shfl_xor_sync(0xffffffffu, r[0], sh);
                }
                // lanes with bit 4 clear hold s^T k, the others s^T q, of column `at`
                const int at = NC == 1 ? 0 : (lane >> 1) & 1;
                const float other = __shfl_xor_sync(0xffffffffu, r[0], 4);
                const float u = sc.y * (st.v[t][cl + at] - ((lane & 4) ? other : r[0]));
                if ((lane & 4) && !(lane & 1) && (NC == 2 || !(lane & 2)) && col + at < d.vdim_p)
                    heads_out[((size_t)(row0 + t0 + t) * d.heads + h) * d.vdim_p + col + at] = fmaf(sc.z, u, r[0]);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float uc = NC == 1 ? u : __shfl_sync(0xffffffffu, u, (lane & 24) | (c << 1));
                    const uint64_t w2 = f32x2(uc, uc);
#pragma unroll
                    for (int m = 0; m < DM * 2; ++m) s[c][m] = fma2(k[m], w2, s[c][m]);
                }
            }
        } else
#pragma unroll 1
        for (int t = 0; t < nt; t += 2) {
            const float4 sc1 = *reinterpret_cast<const float4 *>(st.s[t]), sc2 = *reinterpret_cast<const float4 *>(st.s[t + 1]);
            const float2 cross = *reinterpret_cast<const float2 *>(st.cross[t >> 1]);
            float e1 = 1.0f, e2 = 1.0f, g2 = 1.0f; // decays from the state as held to each token, from the first token to the second
            bool fold = false;                     // the same in every thread of the block
            if constexpr (!CH) {
                g2 = sc2.x;
                fold = G * sc1.x * g2 < 9.5367431640625e-7f;
                if (fold) {
                    rescale(G);
                    G = 1.0f;
                }
                e1 = G * sc1.x;
                e2 = e1 * g2;
            }
            uint64_t k1[DM * 2], k2[DM * 2];
            float r[4 * NC]; // s^T k1, s^T q1, s^T k2, s^T q2, each of the NC columns
            {
                uint64_t acc[4 * NC];
#pragma unroll
                for (int i = 0; i < 4 * NC; ++i) acc[i] = 0ull;
#pragma unroll
                for (int m = 0; m < DM; ++m) {
                    const int at = 32 * m + 4 * part;
                    const ulonglong2 ka = *reinterpret_cast<const ulonglong2 *>(&st.qk[t][1][at]), qa = *reinterpret_cast<const ulonglong2 *>(&st.qk[t][0][at]);
                    const ulonglong2 kb = *reinterpret_cast<const ulonglong2 *>(&st.qk[t + 1][1][at]), qb = *reinterpret_cast<const ulonglong2 *>(&st.qk[t + 1][0][at]);
                    k1[2 * m] = ka.x;
                    k1[2 * m + 1] = ka.y;
                    k2[2 * m] = kb.x;
                    k2[2 * m + 1] = kb.y;
                    ulonglong2 ga, gb;
                    if constexpr (CH) {
                        ga = *reinterpret_cast<const ulonglong2 *>(&st.g[t][at]);
                        gb = *reinterpret_cast<const ulonglong2 *>(&st.g[t + 1][at]);
                        k1[2 * m] = mul2(gb.x, ka.x);
                        k1[2 * m + 1] = mul2(gb.y, ka.y);
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e) { // the accumulators in turn: no sum waits for the one before
                        const uint64_t kae = e ? ka.y : ka.x, qae = e ? qa.y : qa.x, kbe = e ? kb.y : kb.x, qbe = e ? qb.y : qb.x;
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            if constexpr (CH) s[c][2 * m + e] = mul2(e ? ga.y : ga.x, s[c][2 * m + e]);
                            acc[c] = fma2(s[c][2 * m + e], kae, acc[c]);
                            acc[NC + c] = fma2(s[c][2 * m + e], qae, acc[NC + c]);
                        }
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            if constexpr (CH) s[c][2 * m + e] = mul2(e ? gb.y : gb.x, s[c][2 * m + e]);
                            acc[2 * NC + c] = fma2(s[c][2 * m + e], kbe, acc[2 * NC + c]);
                            acc[3 * NC + c] = fma2(s[c][2 * m + e], qbe, acc[3 * NC + c]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 4 * NC; ++i) {
                    const float2 a = f32x2_parts(acc[i]);
                    r[i] = a.x + a.y;
                }
            }
            // reduction over the lanes of the group: halve the values while there are several, then plain
#pragma unroll
            for (int sh = 4, w = 2 * NC; sh; sh >>= 1, w >>= 1) {
                const bool up = (lane & sh) != 0;
#pragma unroll
                for (int i = 0; i < w; ++i) {
                    const float send = up ? r[i] : r[i + w], keep = up ? r[i + w] : r[i];
                    r[i] = keep + __shfl_xor_sync(0xffffffffu, send, sh);
                }
                if (w == 0) r[0] += __shfl_xor_sync(0xffffffffu, r[0], sh);
            }
            float u1[NC], u2[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float a1 = __shfl_sync(0xffffffffu, r[0], (lane & 24) | c), a2 = __shfl_sync(0xffffffffu, r[0], (lane & 24) | 4 | c);
                u1[c] = sc1.y * fmaf(-e1, a1, st.v[t][cl + c]);
                u2[c] = sc2.y * fmaf(-g2 * cross.x, u1[c], fmaf(-e2, a2, st.v[t + 1][cl + c]));
            }
            {
                const bool second = type & 2;
                const float p1 = mine ? u1[NC - 1] : u1[0], p2 = mine ? u2[NC - 1] : u2[0];
                const float out = second ? fmaf(sc2.z, p2, fmaf(g2 * cross.y, p1, e2 * r[0])) : fmaf(sc1.z, p1, e1 * r[0]);
                if (writer && t + (type >> 1) < nt) *o = out;
                o += 2 * o_step;
            }
            float f1 = 1.0f, f2 = 1.0f;
            if constexpr (!CH) {
                if (fold) {
                    rescale(e2);
                    f1 = g2;
                } else {
                    G = e2;
                    f1 = __fdividef(1.0f, e1);
                    f2 = __fdividef(1.0f, e2);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const uint64_t w1 = f32x2(f1 * u1[c], f1 * u1[c]), w2 = f32x2(f2 * u2[c], f2 * u2[c]);
#pragma unroll
                for (int m = 0; m < DM * 2; ++m) s[c][m] = fma2(k2[m], w2, fma2(k1[m], w1, s[c][m]));
            }
        }
        if (tid >= one) stages[b ^ 1].s[st_t][st_j] = next;
        __syncthreads();
        if (*(volatile int *)&abort_flag) { // a copy did not come: reported; leave once this stage's and the next one's are through
            if (tid == 0)
                for (int i = t0 / TOK; i <= t0 / TOK + 1 && i * TOK < n; ++i) tc::mbar_drain(tc::smem_u32(&full[i & 1]), i >> 1 & 1);
            return;
        }
    }
    if (!CH) rescale(G);
#pragma unroll
    for (int m = 0; m < DM; ++m)
#pragma unroll
        for (int e = 0; e < 4; e += 2) {
            const int i = 32 * m + 4 * part + e;
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (i < d.dim_p && col + c < d.vdim_p) {
                    const float2 v = f32x2_parts(s[c][2 * m + e / 2]);
                    S[(size_t)i * d.vdim_p + c] = v.x;
                    S[(size_t)(i + 1) * d.vdim_p + c] = v.y;
                }
        }
    if (cg == 0) {
        float *cring = conv_state + (size_t)slot * d.taps * cw;
        for (int t = max(0, n - d.taps); t < n; ++t) {
            const float *p = proj + (size_t)(row0 + t) * ldp;
            float *c = cring + (size_t)((past + t) % d.taps) * cw;
            if (h % group == 0)
                for (int j = tid; j < d.dim_p; j += T) {
                    c[d.q_at() + kh * d.dim_p + j] = p[d.q_at() + kh * d.dim_p + j];
                    c[d.k_at() + kh * d.dim_p + j] = p[d.k_at() + kh * d.dim_p + j];
                }
            for (int j = tid; j < d.vdim_p; j += T) c[d.v_at() + h * d.vdim_p + j] = p[d.v_at() + h * d.vdim_p + j];
        }
    }
}

// One warp per (row, head).
template <bool CH, typename T>
__global__ void __launch_bounds__(256)
delta_out_kernel(DeltaDims d, Fresh<float> gates, int ldg, const float *__restrict__ norm, Fresh<float> heads_out,
                 int n_rows, T *__restrict__ out) {
    pdl_trigger();
    pdl_wait();
    const int unit = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (unit >= n_rows * d.heads) return;
    const int row = unit / d.heads, h = unit - row * d.heads;
    const Fresh<float> o = heads_out + (size_t)unit * d.vdim_p, g = gates + ((size_t)row * ldg + h * d.vdim_p);
    auto act = [](float z) { return CH ? sigmoid_f(z) : silu_f(z); };
    float4 v[2]; // the first 256 columns stay in registers
    float s = 0.0f;
#pragma unroll
    for (int c = 0; c < 2; ++c) { // columns past vdim hold zeros
        const int j = lane * 4 + 128 * c;
        v[c] = j < d.vdim_p ? o.four(j) : make_float4(0.f, 0.f, 0.f, 0.f);
        s += (v[c].x * v[c].x + v[c].y * v[c].y) + (v[c].z * v[c].z + v[c].w * v[c].w);
    }
    for (int j = 256 + lane; j < d.vdim_p; j += 32) {
        const float t = o[j];
        s = fmaf(t, t, s);
    }
    const float rn = 1.0f / sqrtf(warp_sum(s) / (float)d.vdim + d.eps);
    T *y = out + (size_t)unit * d.vdim_p;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int j = lane * 4 + 128 * c;
        if (j >= d.vdim_p) continue;
        const float4 gg = g.four(j);
        const float e[4] = {v[c].x * act(gg.x), v[c].y * act(gg.y), v[c].z * act(gg.z), v[c].w * act(gg.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) store_from_float(y + j + i, j + i < d.vdim ? e[i] * rn * norm[j + i] : 0.0f);
    }
    for (int j = 256 + lane; j < d.vdim; j += 32) store_from_float(y + j, o[j] * rn * norm[j] * act(g[j]));
}

template <bool CH, typename T>
int step_launch(b200nn_ctx *ctx, const DeltaDims &d, const float *proj, int ldp, const float *ext, const DeltaWeights &w, float *conv_state, float *state,
                const RowMap &rows, int n_rows, T *out) {
    const dim3 grid(d.heads, n_rows);
    const size_t smem = (2 * d.dim_p + 3 * d.vdim_p + 2048 + 8 + (CH ? d.dim_p : 0)) * sizeof(float);
#define DSTEP(R)                                                                                                             \
    do {                                                                                                                     \
        PREFER_SMEM_ONCE((delta_step_kernel<R, CH, T>));                                                                     \
        launch_pdl(ctx, delta_step_kernel<R, CH, T>, grid, dim3(256), smem, d, proj, ldp, ext, w, conv_state, state, rows,   \
                   out);                                                                                                     \
    } while (0)
    if (d.dim_p <= 64) DSTEP(8);
    else if (d.dim_p <= 128) DSTEP(16);
    else DSTEP(32);
#undef DSTEP
    CK_LAUNCH(ctx, "delta_step_kernel");
    return B200NN_OK;
}

// [rows][parts][vectors][width] of f32 rows `ld` apart; a box holds SCAN_TOKENS rows of `box` entries of one vector of every part
int map_rows(b200nn_ctx *ctx, CUtensorMap *map, const float *base, int width, int vectors, int parts, int rows, int ld, int box) {
    if (!ctx->encode_tiled) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is unavailable");
    auto encode = reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(ctx->encode_tiled);
    const cuuint64_t dims[4] = {(cuuint64_t)width, (cuuint64_t)vectors, (cuuint64_t)parts, (cuuint64_t)rows};
    const cuuint64_t strides[3] = {(cuuint64_t)width * 4, (cuuint64_t)width * vectors * 4, (cuuint64_t)ld * 4};
    const cuuint32_t boxes[4] = {(cuuint32_t)box, 1, (cuuint32_t)parts, (cuuint32_t)SCAN_TOKENS}, steps[4] = {1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(base), dims, strides, boxes, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(ctx, B200NN_ERR_CUDA, "cuTensorMapEncodeTiled (delta rule) failed: " + std::to_string((int)r));
    return B200NN_OK;
}

template <bool CH>
int prompt_launch(b200nn_ctx *ctx, const DeltaDims &d, bool b16, const float *proj, int ldp, const float *ext, const DeltaWeights &w, float *conv_state,
                  float *state, const RowMap &rows, const SeqMap &sm, int n_rows, const int *row_seq, float *conv, float *heads_out, void *out) {
    const dim3 cgrid(d.kv_heads + d.heads, (n_rows + 8 * CONV_ROWS - 1) / (8 * CONV_ROWS));
    PREFER_SMEM_ONCE((delta_conv_kernel<1, CH>));
    PREFER_SMEM_ONCE((delta_conv_kernel<2, CH>));
    if (d.dim_p <= 128)
        launch_ordered(ctx, delta_conv_kernel<1, CH>, cgrid, dim3(256), 0, d, proj, ldp, ext, w, conv_state, rows, sm, row_seq, n_rows, conv);
    else
        launch_ordered(ctx, delta_conv_kernel<2, CH>, cgrid, dim3(256), 0, d, proj, ldp, ext, w, conv_state, rows, sm, row_seq, n_rows, conv);
    CK_LAUNCH(ctx, "delta_conv_kernel");
    // columns per lane: one (shorter chains, more instructions) while that gives an SM no more than three blocks; 512 tokens,
    // 8 heads of 128, one / two columns, us: 2 sequences 112 / 119, 4 149 / 126, 8 213 / 168, 16 404 / 267.  Decays per channel cost a
    // multiplication per entry and column and no reduction: three blocks up to a dim of 64, two up to 96, one above (8 heads, 250
    // tokens: dim 128 1 sequence 55 / 61, 2 64.6 / 61.5, 3 77.8 / 67.5; dim 96 2 54 / 55, 3 63.7 / 59.7; dim 64 2 45 / 51, 4 61 / 54).
    const long long columns = (long long)d.vdim_p * d.heads * sm.n_seq;
    const int dm = (d.dim_p + 31) / 32;
    const int blocks = CH ? std::min(3, std::max(1, 5 - dm)) : 3;
    const int nc = dm > 4 ? 1 : ctx->delta_cols ? ctx->delta_cols : columns > 8LL * blocks * ctx->sm_count ? 2 : 1;
    // decays per channel: tokens one at a time (two columns a lane) in passes of a few tokens, where a pair's cross products are most of
    // the work, and for heads of more than 96 in passes that fill the GPU several times over, where its longer chains hide nothing.
    // In pairs / one at a time, us: 128 sequences of 1 40.8 / 34.7, 32 of 3 18.0 / 15.9, 4 of 3 7.3 / 7.1, of 6 8.5 / 8.6; 8 heads of 128, 8
    // sequences of 50 27.3 / 27.7, 12 34.8 / 34.3, 16 41.6 / 40.1, 64 140 / 138; 8 heads of 64, 64 sequences of 50 86.8 / 89.6
    const bool pairs = !CH || !(sm.max_n <= 3 || (dm == 4 && columns > 8LL * 10 * ctx->sm_count));
    CUtensorMap map_qk, map_v, map_g;
    const int dp = dm <= 4 ? dm * 32 : dm <= 6 ? 192 : 256;
    if (int e = map_rows(ctx, &map_qk, conv + d.q_at(), d.dim_p, d.kv_heads, 2, n_rows, d.conv_ld(), dp)) return e;
    if (int e = map_rows(ctx, &map_v, conv + d.v_at(), d.vdim_p, d.heads, 1, n_rows, d.conv_ld(), nc == 1 ? 8 : 16)) return e;
    map_g = map_v; // not read
    if (CH)
        if (int e = map_rows(ctx, &map_g, conv + d.decay_at(), d.dim_p, d.heads, 1, n_rows, d.conv_ld(), dp)) return e;
#define DSCAN(M, C, P)                                                                                                        \
    do {                                                                                                                      \
        constexpr size_t smem = 2 * sizeof(ScanStage<M, C, CH>) + 128;                                                            \
        static bool done[16] = {};                                                                                            \
        if (!done[ctx->device & 15]) {                                                                                        \
            CK(ctx, cudaFuncSetAttribute(delta_scan_kernel<M, C, CH, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
            prefer_max_smem(delta_scan_kernel<M, C, CH, P>);                                                                     \
            done[ctx->device & 15] = true;                                                                                    \
        }                                                                                                                     \
        CK(ctx, launch_ordered(ctx, delta_scan_kernel<M, C, CH, P>, dim3((d.vdim_p + 8 * C - 1) / (8 * C), d.heads, sm.n_seq), \
                               dim3(SCAN_THREADS), smem, map_qk, map_v, map_g, d, proj, ldp, conv, conv_state, state, sm, heads_out, ctx->dev_err));            \
    } while (0)
#define DSCAN_C(M)                                                                                                            \
    do {                                                                                                                      \
        if (CH && nc == 2 && !pairs) DSCAN(M, 2, !CH);                                                                        \
        else if (nc == 2) DSCAN(M, 2, true);                                                                                  \
        else DSCAN(M, 1, true);                                                                                                     \
    } while (0)
    if (dm <= 1) DSCAN_C(1);
    else if (dm <= 2) DSCAN_C(2);
    else if (dm <= 3) DSCAN_C(3);
    else if (dm <= 4) DSCAN_C(4);
    else if (dm <= 6) DSCAN(6, 1, true);
    else DSCAN(8, 1, true);
#undef DSCAN_C
#undef DSCAN
    CK_LAUNCH(ctx, "delta_scan_kernel");
    const int units = n_rows * d.heads;
    const float *gates = CH ? ext + d.ext() : proj + d.g_at();
    const int ldg = CH ? 2 * d.ext() : ldp;
    if (b16) {
        PREFER_SMEM_ONCE((delta_out_kernel<CH, __nv_bfloat16>));
        launch_pdl(ctx, delta_out_kernel<CH, __nv_bfloat16>, dim3((units + 7) / 8), dim3(256), 0, d, gates, ldg, w.norm, heads_out, n_rows,
                   (__nv_bfloat16 *)out);
    } else {
        PREFER_SMEM_ONCE((delta_out_kernel<CH, float>));
        launch_pdl(ctx, delta_out_kernel<CH, float>, dim3((units + 7) / 8), dim3(256), 0, d, gates, ldg, w.norm, heads_out, n_rows, (float *)out);
    }
    CK_LAUNCH(ctx, "delta_out_kernel");
    return B200NN_OK;
}

}  // namespace

int launch_delta_step(b200nn_ctx *ctx, const DeltaDims &d, bool b16, const float *proj, int ldp, const float *ext, const DeltaWeights &w, float *conv_state,
                      float *state, const RowMap &rows, int n_rows, void *out) {
    if (n_rows > 65535) return set_error(ctx, B200NN_ERR_SHAPE, "delta rule: more than 65535 rows");
    if (d.dim_p > 256) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "delta rule: dim > 256");
    if (d.channel)
        return b16 ? step_launch<true>(ctx, d, proj, ldp, ext, w, conv_state, state, rows, n_rows, (__nv_bfloat16 *)out)
                   : step_launch<true>(ctx, d, proj, ldp, ext, w, conv_state, state, rows, n_rows, (float *)out);
    return b16 ? step_launch<false>(ctx, d, proj, ldp, ext, w, conv_state, state, rows, n_rows, (__nv_bfloat16 *)out)
               : step_launch<false>(ctx, d, proj, ldp, ext, w, conv_state, state, rows, n_rows, (float *)out);
}

int launch_delta_prompt(b200nn_ctx *ctx, const DeltaDims &d, bool b16, const float *proj, int ldp, const float *ext, const DeltaWeights &w,
                        float *conv_state, float *state, const RowMap &rows, const SeqMap &sm, int n_rows, const int *row_seq, float *conv,
                        float *heads_out, void *out) {
    if (d.dim_p > 256) return set_error(ctx, B200NN_ERR_UNSUPPORTED, "delta rule: dim > 256");
    if (n_rows > 8 * 65535 || sm.n_seq > 65535) return set_error(ctx, B200NN_ERR_SHAPE, "delta rule: too many rows or sequences in a pass");
    if (ldp & 3) return set_error(ctx, B200NN_ERR_SHAPE, "delta rule: projection rows must keep 16-byte alignment");
    return d.channel ? prompt_launch<true>(ctx, d, b16, proj, ldp, ext, w, conv_state, state, rows, sm, n_rows, row_seq, conv, heads_out, out)
                     : prompt_launch<false>(ctx, d, b16, proj, ldp, ext, w, conv_state, state, rows, sm, n_rows, row_seq, conv, heads_out, out);
}
