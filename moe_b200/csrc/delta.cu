// The gated delta rule: a recurrent mixer whose state is corrected towards each token's value.
//
// Per value head h (query/key head h / (heads / kv_heads)), with a state S [d, dv] that starts at zero:
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//
//   delta_prepare   from the 32-bit projection row [q heads | k heads | v heads | ... | b | a ...]: a causal
//                   convolution over time on every channel of q, k and v (the last taps - 1 rows a
//                   sequence has seen are its state, oldest first) and silu; query and key heads divided
//                   by sqrt(sum(x^2) + eps), queries also times d^(-1/2); per value head
//                   beta = sigmoid(b) and the logarithm of the decay, -exp(A_log) softplus(a + dt_bias).
//                   In a step of one token a sequence the same launch moves the convolution's state on.
//   delta_step      one token a sequence: the recurrence with the state read once and written once, and
//                   the output's norm and gate behind it, a block a (head, sequence).
//   delta_scan      several tokens a sequence, four at a time, the state in registers.
//   delta_chunk, delta_chunk_scan   the same for few long sequences: chunks of sixteen tokens, first what needs no state for
//                   all of them side by side, then the state's way through them.
// The decay g is one number a value head, or one a value head and key channel (the rows of S then shrink each by their
// own): delta_prepare forms those from a product's rows of their own, g = exp(-exp(A_log_h) softplus(a + dt_bias)).
// Everything here is 32-bit arithmetic (delta_chunk's in 64 bits, its results in 32); only the normed, gated output of delta_step
// is rounded.
#include "common.cuh"

namespace {

constexpr int DP_WARPS = 8;
constexpr int DP_MAX_D = 256;

__device__ __forceinline__ float silu32(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_dt(float z) { return z > 20.f ? z : log1pf(expf(z)); }

struct DeltaPrep {
    const float* proj;         // [T, ld]: q (G d), k (G d), v (H dv) from column 0; b and a from columns b_at, a_at
    long long ld;
    int b_at, a_at;
    const float* taps_w;       // [taps, channels]
    float* state;              // per slot (taps - 1) * channels floats, oldest row first
    long long state_pitch;
    const float* a_log;        // [H]
    const float* dt_bias;      // [H]
    const int* seq_of_token;
    const int* cu_seqlens;
    const int* slots;
    int num_tokens, taps, H, G, d, dv, shift;
    float eps, q_scale;
    float* out;                // [T, channels]: q, k, v
    float* step;               // [T, 2 H]: beta, logarithm of the decay
    // decays of a channel (decay not null): a's rows, [T, lda] with H * d columns; dt_bias is [H * d]
    const float* a_rows;
    long long lda;
    float* decay;              // [T, H * d]: the decays themselves
};

// W neighbouring channels of row t convolved and passed through silu; `st`: the sequence's state, li: the row's place
// among the sequence's rows of the step.  With `shift` (one row a sequence) the state's rows move one place down.
template <int W, int TAPS>
__device__ __forceinline__ void conv_silu(const DeltaPrep& p, int t, int li, float* st, int ch, int channels, float* y) {
    const int taps = TAPS > 0 ? TAPS : p.taps;
#pragma unroll
    for (int e = 0; e < W; e++) y[e] = 0.f;
#pragma unroll
    for (int j = 0; j < taps; j++) {
        const int r = li - (taps - 1) + j;
        const float* src = r >= 0 ? p.proj + (size_t)(t - li + r) * p.ld + ch : st + (size_t)(taps - 1 + r) * channels + ch;
        const float* wj = p.taps_w + (size_t)j * channels + ch;
        if (W == 4) {
            const float4 x = *reinterpret_cast<const float4*>(src), w = *reinterpret_cast<const float4*>(wj);
            y[0] = fmaf(w.x, x.x, y[0]), y[1] = fmaf(w.y, x.y, y[1]), y[2] = fmaf(w.z, x.z, y[2]), y[3] = fmaf(w.w, x.w, y[3]);
            if (p.shift && j >= 1) *reinterpret_cast<float4*>(st + (size_t)(j - 1) * channels + ch) = x;
        } else {
            const float x = *src;
            y[0] = fmaf(*wj, x, y[0]);
            if (p.shift && j >= 1) st[(size_t)(j - 1) * channels + ch] = x;
        }
    }
#pragma unroll
    for (int e = 0; e < W; e++) y[e] = silu32(y[e]);
}

// grid (token, parts of its heads); a warp takes one head of q or k, or one run of 32 W channels of v, in turn.
template <int W, int TAPS>
__global__ void __launch_bounds__(DP_WARPS * 32)
delta_prepare_kernel(const DeltaPrep p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x;
    const int qk = 2 * p.G * p.d, channels = qk + p.H * p.dv;
    const int vruns = (p.H * p.dv + 32 * W - 1) / (32 * W);
    const int druns = p.decay ? (p.H * p.d + 32 * W - 1) / (32 * W) : 0;
    const int items = 2 * p.G + vruns + 1 + druns;
    pdl_sync();
    const int s = p.seq_of_token[t];
    float* out = p.out + (size_t)t * channels;
    float* stp = p.step + (size_t)t * 2 * p.H;
    const int li = s >= 0 ? t - p.cu_seqlens[s] : 0;
    float* st = (s >= 0 && p.taps > 1) ? p.state + (size_t)p.slots[s] * p.state_pitch : nullptr;
    for (int item = blockIdx.y * DP_WARPS + warp; item < items; item += gridDim.y * DP_WARPS) {
        if (s < 0) {           // a row of no sequence: something finite, no state touched
            if (item < 2 * p.G) {
                for (int e = lane; e < p.d; e += 32) out[item * p.d + e] = 0.f;
            } else if (item < 2 * p.G + vruns) {
                for (int e = (item - 2 * p.G) * 32 * W + lane; e < min(p.H * p.dv, (item - 2 * p.G + 1) * 32 * W); e += 32)
                    out[qk + e] = 0.f;
            } else if (item == 2 * p.G + vruns) {
                for (int h = lane; h < 2 * p.H; h += 32) stp[h] = 0.f;
            } else {
                const int r0 = (item - 2 * p.G - vruns - 1) * 32 * W;
                for (int e = r0 + lane; e < min(p.H * p.d, r0 + 32 * W); e += 32) p.decay[(size_t)t * p.H * p.d + e] = 1.f;
            }
            continue;
        }
        if (item < 2 * p.G) {
            const int ch0 = item * p.d;
            constexpr int PASSES = DP_MAX_D / (32 * W);
            float y[PASSES][W];
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < PASSES; i++) {
                const int e = (i * 32 + lane) * W;
                if (e < p.d) {
                    conv_silu<W, TAPS>(p, t, li, st, ch0 + e, channels, y[i]);
#pragma unroll
                    for (int z = 0; z < W; z++) ss = fmaf(y[i][z], y[i][z], ss);
                }
            }
            ss = warp_sum(ss);
            float inv = 1.0f / sqrtf(ss + p.eps);
            if (item < p.G) inv *= p.q_scale;
#pragma unroll
            for (int i = 0; i < PASSES; i++) {
                const int e = (i * 32 + lane) * W;
                if (e < p.d) {
                    if (W == 4)
                        *reinterpret_cast<float4*>(out + ch0 + e) =
                            make_float4(y[i][0] * inv, y[i][1 % W] * inv, y[i][2 % W] * inv, y[i][3 % W] * inv);
                    else
                        out[ch0 + e] = y[i][0] * inv;
                }
            }
        } else if (item < 2 * p.G + vruns) {
            const int e = ((item - 2 * p.G) * 32 + lane) * W;
            if (e < p.H * p.dv) {
                float y[W];
                conv_silu<W, TAPS>(p, t, li, st, qk + e, channels, y);
                if (W == 4)
                    *reinterpret_cast<float4*>(out + qk + e) = make_float4(y[0], y[1 % W], y[2 % W], y[3 % W]);
                else
                    out[qk + e] = y[0];
            }
        } else if (item == 2 * p.G + vruns) {
            const float* row = p.proj + (size_t)t * p.ld;
            for (int h = lane; h < p.H; h += 32) {
                stp[h] = 1.0f / (1.0f + expf(-row[p.b_at + h]));
                stp[p.H + h] = p.decay ? 0.f : -expf(p.a_log[h]) * softplus_dt(row[p.a_at + h] + p.dt_bias[h]);
            }
        } else {
            const int e = ((item - 2 * p.G - vruns - 1) * 32 + lane) * W;
            if (e < p.H * p.d) {
                const float* a = p.a_rows + (size_t)t * p.lda + e;
                const float rate = expf(p.a_log[e / p.d]);            // (W neighbours lie in one head)
                float* dst = p.decay + (size_t)t * p.H * p.d + e;
                if (W == 4) {
                    const float4 x = *reinterpret_cast<const float4*>(a), b = *reinterpret_cast<const float4*>(p.dt_bias + e);
                    *reinterpret_cast<float4*>(dst) = make_float4(expf(-rate * softplus_dt(x.x + b.x)), expf(-rate * softplus_dt(x.y + b.y)),
                                                                  expf(-rate * softplus_dt(x.z + b.z)), expf(-rate * softplus_dt(x.w + b.w)));
                } else {
                    *dst = expf(-rate * softplus_dt(*a + p.dt_bias[e]));
                }
            }
        }
    }
}

// The same for many tokens, four channels a lane, heads of up to 128: a warp takes one item of a RUN of tokens, whose rows it reads once (a
// row is read by the tokens of its own run and by one more for its last taps - 1, not by TAPS blocks; a channel's taps once a run, not
// once a token).  Sums in the order of the kernel above, so the results are the same to the bit.  2,048 tokens, 16 heads of 128: 70 -> 50 us.
constexpr int DP_RUN = 8;
template <int TAPS>
__global__ void __launch_bounds__(DP_WARPS * 32, 3)
delta_prepare_run_kernel(const DeltaPrep p) {
    __shared__ int s_seq[DP_RUN], s_li[DP_RUN];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = blockIdx.x * DP_RUN, n = min(DP_RUN, p.num_tokens - t0);
    const int qk = 2 * p.G * p.d, channels = qk + p.H * p.dv;
    const int vruns = (p.H * p.dv + 127) / 128, druns = p.decay ? (p.H * p.d + 127) / 128 : 0;
    const int items = 2 * p.G + vruns + 1 + druns;
    pdl_sync();
    if (threadIdx.x < DP_RUN) {
        const int t = t0 + threadIdx.x, s = threadIdx.x < n ? p.seq_of_token[t] : -1;
        s_seq[threadIdx.x] = s, s_li[threadIdx.x] = s >= 0 ? t - p.cu_seqlens[s] : 0;
    }
    __syncthreads();
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int item = blockIdx.y * DP_WARPS + warp; item < items; item += gridDim.y * DP_WARPS) {
        if (item < 2 * p.G + vruns) {
            const bool head = item < 2 * p.G;
            const int e = head ? lane * 4 : (item - 2 * p.G) * 128 + lane * 4, ch = (head ? item * p.d : qk) + e;
            const bool on = e < (head ? p.d : p.H * p.dv);
            float4 w[TAPS], x[DP_RUN], win[TAPS - 1];
#pragma unroll
            for (int j = 0; j < TAPS; j++) w[j] = on ? *reinterpret_cast<const float4*>(p.taps_w + (size_t)j * channels + ch) : zero;
#pragma unroll
            for (int i = 0; i < DP_RUN; i++)
                x[i] = on && i < n ? *reinterpret_cast<const float4*>(p.proj + (size_t)(t0 + i) * p.ld + ch) : zero;
#pragma unroll
            for (int j = 0; j < TAPS - 1; j++) win[j] = zero;
            int before = -1;
#pragma unroll
            for (int i = 0; i < DP_RUN; i++) {
                if (i >= n) break;
                const int s = s_seq[i];
                float* out = p.out + (size_t)(t0 + i) * channels + ch;
                if (s < 0) {               // a row of no sequence: something finite, no state touched
                    if (on) *reinterpret_cast<float4*>(out) = zero;
                    before = -1;
                    continue;
                }
                if (s != before) {         // the rows before this one: the step's, or the sequence's state
                    const int li = s_li[i];
                    const float* st = p.state + (size_t)p.slots[s] * p.state_pitch;
#pragma unroll
                    for (int j = 0; j < TAPS - 1; j++) {
                        const int r = li - (TAPS - 1) + j;
                        if (on) win[j] = *reinterpret_cast<const float4*>(r >= 0 ? p.proj + (size_t)(t0 + i - li + r) * p.ld + ch
                                                                                 : st + (size_t)(TAPS - 1 + r) * channels + ch);
                    }
                    before = s;
                }
                float4 y = zero;
#pragma unroll
                for (int j = 0; j < TAPS; j++) {
                    const float4 v = j < TAPS - 1 ? win[j < TAPS - 1 ? j : 0] : x[i];
                    y.x = fmaf(w[j].x, v.x, y.x), y.y = fmaf(w[j].y, v.y, y.y), y.z = fmaf(w[j].z, v.z, y.z), y.w = fmaf(w[j].w, v.w, y.w);
                }
#pragma unroll
                for (int j = 0; j < TAPS - 1; j++) win[j] = j < TAPS - 2 ? win[j + 1 < TAPS - 1 ? j + 1 : 0] : x[i];
                y = make_float4(silu32(y.x), silu32(y.y), silu32(y.z), silu32(y.w));
                if (head) {
                    float ss = 0.f;
                    if (on) ss = fmaf(y.x, y.x, ss), ss = fmaf(y.y, y.y, ss), ss = fmaf(y.z, y.z, ss), ss = fmaf(y.w, y.w, ss);
                    ss = warp_sum(ss);
                    float inv = 1.0f / sqrtf(ss + p.eps);
                    if (item < p.G) inv *= p.q_scale;
                    y = make_float4(y.x * inv, y.y * inv, y.z * inv, y.w * inv);
                }
                if (on) *reinterpret_cast<float4*>(out) = y;
            }
        } else if (item == 2 * p.G + vruns) {
            for (int i = 0; i < n; i++) {
                const float* row = p.proj + (size_t)(t0 + i) * p.ld;
                float* stp = p.step + (size_t)(t0 + i) * 2 * p.H;
                const bool live = s_seq[i] >= 0;
                for (int h = lane; h < p.H; h += 32) {
                    stp[h] = live ? 1.0f / (1.0f + expf(-row[p.b_at + h])) : 0.f;
                    stp[p.H + h] = live && !p.decay ? -expf(p.a_log[h]) * softplus_dt(row[p.a_at + h] + p.dt_bias[h]) : 0.f;
                }
            }
        } else {
            const int e = ((item - 2 * p.G - vruns - 1) * 32 + lane) * 4;
            if (e >= p.H * p.d) continue;
            const float rate = expf(p.a_log[e / p.d]);                // (four neighbours lie in one head)
            const float4 b = *reinterpret_cast<const float4*>(p.dt_bias + e);
            float4 x[DP_RUN];
#pragma unroll
            for (int i = 0; i < DP_RUN; i++) x[i] = i < n ? *reinterpret_cast<const float4*>(p.a_rows + (size_t)(t0 + i) * p.lda + e) : zero;
#pragma unroll
            for (int i = 0; i < DP_RUN; i++) {
                if (i >= n) break;
                float4* dst = reinterpret_cast<float4*>(p.decay + (size_t)(t0 + i) * p.H * p.d + e);
                *dst = s_seq[i] < 0 ? make_float4(1.f, 1.f, 1.f, 1.f)
                                    : make_float4(expf(-rate * softplus_dt(x[i].x + b.x)), expf(-rate * softplus_dt(x[i].y + b.y)),
                                                  expf(-rate * softplus_dt(x[i].z + b.z)), expf(-rate * softplus_dt(x[i].w + b.w)));
            }
        }
    }
}

struct DeltaSeq {
    const float* qkv;          // [T, channels] prepared q, k, v
    const float* step;         // [T, 2 H]
    float* state;              // per slot H * d * dv floats ([head][d][dv]) from the pointer given
    long long state_pitch;
    const int* cu_seqlens;
    const int* slots;
    int H, G, d, dv;
    const float* decay;        // [T, H d]: a decay a channel; null: one a head (step)
};

// ---- one token a sequence --------------------------------------------------------------------------
// A block a (head, sequence): thread (cg, kp) holds four neighbouring columns of every KP-th row of S.  The
// state is asked for before the wait for the predecessor: nothing since the step before has written it.
template <typename OT, int UNITS, bool CH>
__global__ void __launch_bounds__(256)
delta_step_kernel(const DeltaSeq p, const float* __restrict__ gate, long long ldg, const float* __restrict__ norm_w,
                  float norm_eps, const int* __restrict__ seq_of_token, int num_tokens, int gate_fn, OT* __restrict__ out) {
    extern __shared__ __align__(16) float ds_smem[];         // k [d] | q [d] | u [dv] | parts [KP][dv] | CH: decays [d]
    __shared__ float red[32];
    const int h = blockIdx.x, s = blockIdx.y, d = p.d, dv = p.dv;
    const int CG = dv / 4, KP = blockDim.x / CG, cg = threadIdx.x % CG, kp = threadIdx.x / CG;
    const bool worker = kp < KP;
    float* sk = ds_smem;
    float* sq = sk + d;
    float* su = sq + d;
    float* parts = su + dv;
    float* sg = parts + KP * dv;
    const int t = p.cu_seqlens[s];
    const bool live = p.cu_seqlens[s + 1] > t && t < num_tokens && seq_of_token[t] >= 0;
    float* S = p.state + (size_t)p.slots[s] * p.state_pitch + (size_t)h * d * dv;
    float4 r[UNITS];
#pragma unroll
    for (int i = 0; i < UNITS; i++) {
        const int row = kp + i * KP;
        r[i] = (live && worker && row < d) ? *reinterpret_cast<const float4*>(S + (size_t)row * dv + cg * 4)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_sync();
    if (!live) {                                             // row s is a row of no sequence: something finite
        if (s < num_tokens && seq_of_token[s] < 0)
            for (int c = threadIdx.x; c < dv; c += blockDim.x) st_f(out + ((size_t)s * p.H + h) * dv + c, 0.f);
        return;
    }
    const int g = h / (p.H / p.G), channels = 2 * p.G * d + p.H * dv;
    const float* row = p.qkv + (size_t)t * channels;
    for (int i = threadIdx.x; i < d; i += blockDim.x) sq[i] = row[(size_t)g * d + i], sk[i] = row[(size_t)(p.G + g) * d + i];
    if (CH)
        for (int i = threadIdx.x; i < d; i += blockDim.x) sg[i] = p.decay[((size_t)t * p.H + h) * d + i];
    const float beta = p.step[(size_t)t * 2 * p.H + h];
    float decay = CH ? 1.f : expf(p.step[(size_t)t * 2 * p.H + p.H + h]);
    __syncthreads();
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < UNITS; i++) {
        const int rr = kp + i * KP;
        if (CH) decay = (worker && rr < d) ? sg[rr] : 0.f;
        r[i].x *= decay, r[i].y *= decay, r[i].z *= decay, r[i].w *= decay;
        if (worker && rr < d) {
            const float k = sk[rr];
            acc.x = fmaf(k, r[i].x, acc.x), acc.y = fmaf(k, r[i].y, acc.y);
            acc.z = fmaf(k, r[i].z, acc.z), acc.w = fmaf(k, r[i].w, acc.w);
        }
    }
    if (worker) *reinterpret_cast<float4*>(parts + (size_t)kp * dv + cg * 4) = acc;
    __syncthreads();
    for (int c = threadIdx.x; c < dv; c += blockDim.x) {
        float held = 0.f;
        for (int q = 0; q < KP; q++) held += parts[(size_t)q * dv + c];
        su[c] = beta * (row[(size_t)2 * p.G * d + (size_t)h * dv + c] - held);
    }
    __syncthreads();
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (worker) {
        const float4 u = *reinterpret_cast<const float4*>(su + cg * 4);
#pragma unroll
        for (int i = 0; i < UNITS; i++) {
            const int rr = kp + i * KP;
            if (rr < d) {
                const float k = sk[rr], q = sq[rr];
                r[i].x = fmaf(k, u.x, r[i].x), r[i].y = fmaf(k, u.y, r[i].y), r[i].z = fmaf(k, u.z, r[i].z), r[i].w = fmaf(k, u.w, r[i].w);
                acc.x = fmaf(q, r[i].x, acc.x), acc.y = fmaf(q, r[i].y, acc.y);
                acc.z = fmaf(q, r[i].z, acc.z), acc.w = fmaf(q, r[i].w, acc.w);
                *reinterpret_cast<float4*>(S + (size_t)rr * dv + cg * 4) = r[i];
            }
        }
        *reinterpret_cast<float4*>(parts + (size_t)kp * dv + cg * 4) = acc;
    }
    __syncthreads();
    // the output's norm over the head and its gate
    float ss = 0.f;
    for (int c = threadIdx.x; c < dv; c += blockDim.x) {
        float o = 0.f;
        for (int q = 0; q < KP; q++) o += parts[(size_t)q * dv + c];
        su[c] = o;
        ss = fmaf(o, o, ss);
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)dv + norm_eps);
    for (int c = threadIdx.x; c < dv; c += blockDim.x)
        st_f(out + ((size_t)t * p.H + h) * dv + c,
             su[c] * inv * norm_w[(size_t)h * dv + c] * gate_value(gate_fn, gate[(size_t)t * ldg + (size_t)h * dv + c]));
}

// ---- several tokens a sequence: four at a time ------------------------------------------------------------
// With b_i the sum of the decays' logarithms from a group's first token to its i-th, S the state before the group,
// and the index pairs j < i (or j <= i) inside the group,
//     u_i = beta_i v_i - beta_i e^(b_i) S^T k_i - sum_(j<i) beta_i e^(b_i - b_j) (k_i . k_j) u_j
//     o_i = e^(b_i) S^T q_i + sum_(j<=i) e^(b_i - b_j) (q_i . k_j) u_j
//     S   <- e^(b_4) S + sum_j k_j (e^(b_4 - b_j) u_j)^T
// (CH, a decay a channel: with G_i the product of the channel's decays from the group's first token to its i-th and
// D_ij that from the one after j to i, e^(b_i) S^T k_i becomes S^T (G_i k_i), e^(b_i - b_j) (k_i . k_j) the sum over the
// channels of D_ij k_i k_j, and S <- G_4 S + sum_j (D_4j k_j) u_j^T; every factor is a product of decays, none a
// quotient.  The warp that forms a group's scalars puts G_i k_i, G_i q_i and D_4j k_j in the place of k, q and the decays.)
// which is the recurrence written out: every exponent is <= 0, only the order of additions differs.  Against
// one token at a time the products with S are eight independent sums instead of two with an update between
// them, their sums over the threads are formed together, and the state is multiplied by a decay once.
//
// grid (ceil(dv / COLS), heads, sequences), 128 threads: thread (kp = tid % KP, cg = tid / KP) holds four neighbouring
// columns of rows 4 kp ... 4 kp + 3 of every 4 KP rows of S in registers (rows beyond d stay zero; the KP
// threads' reads of a token's k and q are then neighbours in shared memory).  KP = 16 (32 columns a block) or, where those
// blocks would leave SMs idle, 32 (16 columns a block, half as many rows a thread).  A run of sixteen tokens is staged
// in shared memory as [k | q | the block's columns of v] a token (cp.async, two buffers; rows beyond the
// sequence's last token are zeros with beta 0 and decay 1: they change nothing); warp w forms the scalars of the
// run's group w.  Within a run the groups follow one another without a block barrier.
constexpr int DG = 4, DRUN = 16, DTHREADS = 128;
__host__ __device__ constexpr int dcols(int kp) { return 4 * (DTHREADS / kp); }

__device__ __forceinline__ void cp_zfill(float* dst, const float* src, int bytes, bool on) {
    const unsigned at = (unsigned)__cvta_generic_to_shared(dst);
    const int n = on ? bytes : 0;
    if (bytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(at), "l"(src), "r"(n) : "memory");
}

// VEC: rows of q, k and v start on 16-byte boundaries and hold whole 16-byte units.
template <int RPT, int KP, bool CH>
__host__ __device__ constexpr size_t delta_scan_floats() {
    return (size_t)2 * DRUN * ((CH ? 3 : 2) * RPT * KP + dcols(KP)) + 4 * DRUN + 4 * 32 + DG * dcols(KP) + (CH ? 4 * RPT * KP : 0);
}
template <int RPT, int KP, bool VEC, bool CH>
__global__ void __launch_bounds__(DTHREADS, RPT <= 8 ? (CH && RPT == 8 ? 3 : 4) : 2)
delta_scan_kernel(const DeltaSeq p, float* __restrict__ o) {
    constexpr int NP = RPT * KP, DCOLS = dcols(KP);
    constexpr int V_AT = (CH ? 3 : 2) * NP;                   // a token's row: k, q, CH: its decays, then v
    constexpr int ROWLEN = V_AT + DCOLS;
    extern __shared__ __align__(16) float sm[];               // [2][DRUN][ROWLEN] | steps [2][2][DRUN] | scalars [4][32] | u [DG][DCOLS]
    float* s_step = sm + 2 * DRUN * ROWLEN;                   // | CH: a group's decay of a channel [4][NP]
    float* s_coef = s_step + 4 * DRUN;
    float* s_u = s_coef + 4 * 32;
    float* s_g4 = s_u + DG * DCOLS;
    const int tid = threadIdx.x, kp = tid % KP, cg = tid / KP, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y, s = blockIdx.z, g = h / (p.H / p.G), d = p.d, dv = p.dv;
    const int c0 = blockIdx.x * DCOLS, col = c0 + cg * 4;
    for (int i = tid; i < 2 * DRUN * ROWLEN; i += DTHREADS) sm[i] = 0.f;         // columns that no copy writes stay zero
    pdl_sync();
    const int tok0 = p.cu_seqlens[s], cnt = p.cu_seqlens[s + 1] - tok0;
    if (cnt <= 0) return;
    const int channels = 2 * p.G * d + p.H * dv, ncols = min(DCOLS, dv - c0);
    float* S = p.state + (size_t)p.slots[s] * p.state_pitch + (size_t)h * d * dv;
    const bool vec_state = dv % 4 == 0 && ((uintptr_t)S) % 16 == 0;
    float sreg[RPT][4];
#pragma unroll
    for (int m = 0; m < RPT; m++) {
        const int n = (m / 4) * 4 * KP + kp * 4 + m % 4;
        if (vec_state && n < d && col < dv) {
            const float4 t4 = *reinterpret_cast<const float4*>(S + (size_t)n * dv + col);
            sreg[m][0] = t4.x, sreg[m][1] = t4.y, sreg[m][2] = t4.z, sreg[m][3] = t4.w;
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++) sreg[m][c] = (n < d && col + c < dv) ? S[(size_t)n * dv + col + c] : 0.f;
        }
    }
    const float* base = p.qkv + (size_t)tok0 * channels;
    const float* sbase = p.step + (size_t)tok0 * 2 * p.H + h;
    const float* gbase = CH ? p.decay + ((size_t)tok0 * p.H + h) * d : nullptr;
    const int k_at = (p.G + g) * d, q_at = g * d, v_at = 2 * p.G * d + h * dv + c0;
    auto stage = [&](int t0, int buf) {
        float* dst = sm + buf * DRUN * ROWLEN;
        constexpr int W = VEC ? 4 : 1;
        const int kw = d / W, vw = ncols / W, per = 2 * kw + vw + (CH ? kw : 0);
        for (int tt = warp; tt < DRUN; tt += DTHREADS / 32) {           // a warp a token
            const bool on = t0 + tt < cnt;
            const float* row = base + (size_t)min(t0 + tt, cnt - 1) * channels;
            float* to = dst + tt * ROWLEN;
            for (int e = lane; e < per; e += 32) {
                if (CH && e >= 2 * kw + vw) {
                    const int x = e - 2 * kw - vw;
                    cp_zfill(to + 2 * NP + x * W, gbase + (size_t)min(t0 + tt, cnt - 1) * p.H * d + x * W, 4 * W, on);
                    continue;
                }
                const int x = e < kw ? e : e < 2 * kw ? e - kw : e - 2 * kw;
                cp_zfill(to + (e < kw ? 0 : e < 2 * kw ? NP : V_AT) + x * W, row + (e < kw ? k_at : e < 2 * kw ? q_at : v_at) + x * W, 4 * W, on);
            }
        }
        if (tid < 2 * DRUN) {
            const int tt = tid % DRUN, which = tid / DRUN;
            cp_zfill(s_step + (buf * 2 + which) * DRUN + tt, sbase + (size_t)min(t0 + tt, cnt - 1) * 2 * p.H + which * p.H, 4, t0 + tt < cnt);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    __syncthreads();                                  // the zeros are there before any copy writes
    stage(0, 0);
    const bool b0 = (kp & 1) != 0, b1 = (kp & 2) != 0, b2 = (kp & 4) != 0, b3 = (kp & 8) != 0;
    const int my_col = (b0 ? 2 : 0) + (b1 ? 1 : 0);
    for (int t0 = 0, buf = 0; t0 < cnt; t0 += DRUN, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                              // this run is there, and the one before is no longer read
        if (t0 + DRUN < cnt) stage(t0 + DRUN, buf ^ 1);
        float* run = sm + buf * DRUN * ROWLEN;
        {
            // the scalars of group `warp`: products of its keys and queries, then everything made of them
            float* row = run + warp * DG * ROWLEN;
            float dots[16];                           // [0 ... 5] k_i . k_j, j < i;  [6 ... 15] q_i . k_j, j <= i
#pragma unroll
            for (int i = 0; i < 16; i++) dots[i] = 0.f;
            for (int e = lane * 4; e < NP; e += 128) {
                float4 k4[DG], q4[DG];
#pragma unroll
                for (int i = 0; i < DG; i++) {
                    k4[i] = *reinterpret_cast<const float4*>(row + i * ROWLEN + e);
                    q4[i] = *reinterpret_cast<const float4*>(row + i * ROWLEN + NP + e);
                }
                if (CH) {
                    const int left = cnt - t0 - warp * DG;        // tokens of the group; places beyond keep what there is
                    float4 g4[DG];
#pragma unroll
                    for (int i = 0; i < DG; i++)
                        g4[i] = i < left ? *reinterpret_cast<const float4*>(row + i * ROWLEN + 2 * NP + e) : make_float4(1.f, 1.f, 1.f, 1.f);
                    auto mul = [](float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); };
                    auto dot3 = [](float4 a, float4 b, float4 c, float s) {
                        return fmaf(a.x * c.x, b.x, fmaf(a.y * c.y, b.y, fmaf(a.z * c.z, b.z, fmaf(a.w * c.w, b.w, s))));
                    };
                    float4 all = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
                    for (int j = 0; j < DG; j++) {
                        float4 since = make_float4(1.f, 1.f, 1.f, 1.f);        // from the token after j to i
#pragma unroll
                        for (int i = j; i < DG; i++) {
                            if (i > j) since = mul(since, g4[i]), dots[i * (i - 1) / 2 + j] = dot3(k4[i], k4[j], since, dots[i * (i - 1) / 2 + j]);
                            dots[6 + i * (i + 1) / 2 + j] = dot3(q4[i], k4[j], since, dots[6 + i * (i + 1) / 2 + j]);
                        }
                        all = mul(all, g4[j]);
                        *reinterpret_cast<float4*>(row + j * ROWLEN + e) = mul(k4[j], all);
                        *reinterpret_cast<float4*>(row + j * ROWLEN + NP + e) = mul(q4[j], all);
                        *reinterpret_cast<float4*>(row + j * ROWLEN + 2 * NP + e) = mul(k4[j], since);
                    }
                    *reinterpret_cast<float4*>(s_g4 + warp * NP + e) = all;
                    continue;
                }
                int x = 0;
#pragma unroll
                for (int i = 1; i < DG; i++)
#pragma unroll
                    for (int j = 0; j < i; j++, x++)
                        dots[x] = fmaf(k4[i].x, k4[j].x, fmaf(k4[i].y, k4[j].y, fmaf(k4[i].z, k4[j].z, fmaf(k4[i].w, k4[j].w, dots[x]))));
#pragma unroll
                for (int i = 0; i < DG; i++)
#pragma unroll
                    for (int j = 0; j <= i; j++, x++)
                        dots[x] = fmaf(q4[i].x, k4[j].x, fmaf(q4[i].y, k4[j].y, fmaf(q4[i].z, k4[j].z, fmaf(q4[i].w, k4[j].w, dots[x]))));
            }
            // sixteen sums over the warp; lane l ends with number l & 15
            float v8[8], v4[4], v2[2];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const bool up = (lane & 8) != 0;
                v8[i] = (up ? dots[8 + i] : dots[i]) + __shfl_xor_sync(0xffffffffu, up ? dots[i] : dots[8 + i], 8);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const bool up = (lane & 4) != 0;
                v4[i] = (up ? v8[4 + i] : v8[i]) + __shfl_xor_sync(0xffffffffu, up ? v8[i] : v8[4 + i], 4);
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const bool up = (lane & 2) != 0;
                v2[i] = (up ? v4[2 + i] : v4[i]) + __shfl_xor_sync(0xffffffffu, up ? v4[i] : v4[2 + i], 2);
            }
            const bool up = (lane & 1) != 0;
            float dot = (up ? v2[1] : v2[0]) + __shfl_xor_sync(0xffffffffu, up ? v2[0] : v2[1], 1);
            dot += __shfl_xor_sync(0xffffffffu, dot, 16);
            // [0 ... 3] beta_i  [4 ... 7] beta_i e^(b_i)  [8 ... 11] e^(b_i)  [12 ... 15] e^(b_4 - b_i)  [16 ... 21] beta_i e^(b_i - b_j) k_i . k_j
            // [22 ... 31] e^(b_i - b_j) q_i . k_j
            const float* be = s_step + buf * 2 * DRUN + warp * DG;
            const float* lg = be + DRUN;
            const float bs[DG] = {lg[0], lg[0] + lg[1], lg[0] + lg[1] + lg[2], lg[0] + lg[1] + lg[2] + lg[3]};
            const int n = lane & 15;
            if (lane < 16) {
                const int i = n & 3;
                const float ei = CH ? 1.f : expf(i == 0 ? bs[0] : i == 1 ? bs[1] : i == 2 ? bs[2] : bs[3]);
                float rest = 0.f;                     // b_4 - b_i, added up and not subtracted
                for (int e = i + 1; e < DG; e++) rest += lg[e];
                s_coef[warp * 32 + n] = n < 4 ? be[i] : n < 8 ? be[i] * ei : n < 12 ? ei : CH ? 1.f : expf(rest);
            } else {
                // pair number n: j < i of the keys, then j <= i of queries and keys
                const int i = n < 6 ? (n < 1 ? 1 : n < 3 ? 2 : 3) : (n < 7 ? 0 : n < 9 ? 1 : n < 12 ? 2 : 3);
                const int j = n < 6 ? n - i * (i - 1) / 2 : n - 6 - i * (i + 1) / 2;
                float decay = 0.f;                    // b_i - b_j, the same
                for (int e = j + 1; e <= i; e++) decay += lg[e];
                s_coef[warp * 32 + 16 + n] = dot * (CH ? 1.f : expf(decay)) * (n < 6 ? be[i] : 1.f);
            }
        }
        __syncthreads();
        const int groups = (min(DRUN, cnt - t0) + DG - 1) / DG;
        for (int gr = 0; gr < groups; gr++) {
            const float* row = run + gr * DG * ROWLEN + kp * 4;
            float kr[DG][RPT];
            float hk[DG][4], hq[DG][4];
#pragma unroll
            for (int i = 0; i < DG; i++)
#pragma unroll
                for (int c = 0; c < 4; c++) hk[i][c] = 0.f, hq[i][c] = 0.f;
#pragma unroll
            for (int m0 = 0; m0 < RPT; m0 += 4) {
#pragma unroll
                for (int i = 0; i < DG; i++) {
                    const float4 k4 = *reinterpret_cast<const float4*>(row + i * ROWLEN + m0 * KP);
                    const float4 q4 = *reinterpret_cast<const float4*>(row + i * ROWLEN + NP + m0 * KP);
                    kr[i][m0] = k4.x, kr[i][m0 + 1] = k4.y, kr[i][m0 + 2] = k4.z, kr[i][m0 + 3] = k4.w;
                    const float qi[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                    for (int z = 0; z < 4; z++)
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            hk[i][c] = fmaf(kr[i][m0 + z], sreg[m0 + z][c], hk[i][c]);
                            hq[i][c] = fmaf(qi[z], sreg[m0 + z][c], hq[i][c]);
                        }
                }
            }
            // Sums over the threads of a column group.  On the way every thread drops what another one
            // carries on: bits 0 and 1 of kp pick the column, bit 2 the product with the keys or the queries.
            float r2[2 * DG][2], r1[2 * DG], rr[DG];
#pragma unroll
            for (int i = 0; i < DG; i++)
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    r2[i][c] = (b0 ? hk[i][2 + c] : hk[i][c]) + __shfl_xor_sync(0xffffffffu, b0 ? hk[i][c] : hk[i][2 + c], 1);
                    r2[DG + i][c] = (b0 ? hq[i][2 + c] : hq[i][c]) + __shfl_xor_sync(0xffffffffu, b0 ? hq[i][c] : hq[i][2 + c], 1);
                }
#pragma unroll
            for (int i = 0; i < 2 * DG; i++)
                r1[i] = (b1 ? r2[i][1] : r2[i][0]) + __shfl_xor_sync(0xffffffffu, b1 ? r2[i][0] : r2[i][1], 2);
#pragma unroll
            for (int i = 0; i < DG; i++) {
                rr[i] = (b2 ? r1[DG + i] : r1[i]) + __shfl_xor_sync(0xffffffffu, b2 ? r1[i] : r1[DG + i], 4);
                rr[i] += __shfl_xor_sync(0xffffffffu, rr[i], 8);
                if (KP == 32) rr[i] += __shfl_xor_sync(0xffffffffu, rr[i], 16);
            }
            float cf[32];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float4 c4 = *reinterpret_cast<const float4*>(s_coef + gr * 32 + i * 4);
                cf[4 * i] = c4.x, cf[4 * i + 1] = c4.y, cf[4 * i + 2] = c4.z, cf[4 * i + 3] = c4.w;
            }
            // (threads of the queries' half go through the same motions with their own sums; their u is not used)
            float u[DG];
            const float* vrow = run + gr * DG * ROWLEN + V_AT + cg * 4 + my_col;
            u[0] = cf[0] * vrow[0] - cf[4] * rr[0];
            u[1] = cf[1] * vrow[ROWLEN] - cf[5] * rr[1] - cf[16] * u[0];
            u[2] = cf[2] * vrow[2 * ROWLEN] - cf[6] * rr[2] - cf[17] * u[0] - cf[18] * u[1];
            u[3] = cf[3] * vrow[3 * ROWLEN] - cf[7] * rr[3] - cf[19] * u[0] - cf[20] * u[1] - cf[21] * u[2];
#pragma unroll
            for (int i = 0; i < DG; i++) {
                if (!b2 && !b3 && kp < 16) s_u[i * DCOLS + cg * 4 + my_col] = cf[12 + i] * u[i];
                const float other = __shfl_xor_sync(0xffffffffu, u[i], 4);
                u[i] = b2 ? other : u[i];
            }
            __syncwarp();                             // a column group's threads lie in one warp
            if (b2 && !b3 && kp < 16 && col + my_col < dv) {
                const float out[DG] = {cf[8] * rr[0] + cf[22] * u[0], cf[9] * rr[1] + cf[23] * u[0] + cf[24] * u[1],
                                       cf[10] * rr[2] + cf[25] * u[0] + cf[26] * u[1] + cf[27] * u[2],
                                       cf[11] * rr[3] + cf[28] * u[0] + cf[29] * u[1] + cf[30] * u[2] + cf[31] * u[3]};
                const int t = t0 + gr * DG;
#pragma unroll
                for (int i = 0; i < DG; i++)
                    if (t + i < cnt) o[(size_t)(tok0 + t + i) * p.H * dv + (size_t)h * dv + col + my_col] = out[i];
            }
            float uw[DG][4];
#pragma unroll
            for (int i = 0; i < DG; i++) {
                const float4 u4 = *reinterpret_cast<const float4*>(s_u + i * DCOLS + cg * 4);
                uw[i][0] = u4.x, uw[i][1] = u4.y, uw[i][2] = u4.z, uw[i][3] = u4.w;
            }
            __syncwarp();                             // read by all before the next group's are written
            if (CH) {                                 // the decays and the keys of the update, row by row
#pragma unroll
                for (int m0 = 0; m0 < RPT; m0 += 4) {
                    const float4 g4 = *reinterpret_cast<const float4*>(s_g4 + gr * NP + kp * 4 + m0 * KP);
                    const float gm[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                    for (int z = 0; z < 4; z++)
#pragma unroll
                        for (int c = 0; c < 4; c++) sreg[m0 + z][c] *= gm[z];
#pragma unroll
                    for (int i = 0; i < DG; i++) {
                        const float4 k4 = *reinterpret_cast<const float4*>(row + i * ROWLEN + 2 * NP + m0 * KP);
                        const float km[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                        for (int z = 0; z < 4; z++)
#pragma unroll
                            for (int c = 0; c < 4; c++) sreg[m0 + z][c] = fmaf(km[z], uw[i][c], sreg[m0 + z][c]);
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < (CH ? 0 : RPT); m++)
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    float x = cf[11] * sreg[m][c];
#pragma unroll
                    for (int i = 0; i < DG; i++) x = fmaf(kr[i][m], uw[i][c], x);
                    sreg[m][c] = x;
                }
        }
    }
#pragma unroll
    for (int m = 0; m < RPT; m++) {
        const int n = (m / 4) * 4 * KP + kp * 4 + m % 4;
        if (n >= d) continue;
        if (vec_state && col < dv) {
            *reinterpret_cast<float4*>(S + (size_t)n * dv + col) = make_float4(sreg[m][0], sreg[m][1], sreg[m][2], sreg[m][3]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (col + c < dv) S[(size_t)n * dv + col + c] = sreg[m][c];
        }
    }
}

// ---- several tokens a sequence: sixteen at a time ---------------------------------------------------------------
// The same recurrence over chunks of sixteen tokens, in two launches.  What does not need the state is formed for all
// chunks side by side (delta_chunk_kernel): with L_ij = beta_i (sum_c D_ij k_i k_j) for j < i, the u of a chunk solve
// (I + L) u = beta (v - (G k) S), so with W = (I + L)^-1 beta (G k), U = (I + L)^-1 beta v (forward substitution, a
// column a thread) and P_ij = sum_c D_ij q_i k_j, j <= i,
//     u = U - W S,    o = (G q) S + P u = Q S + P U with Q = G q - P W,    S <- G_16 S + (D_16 k)^T u
// and the chain over the chunks (delta_chunk_scan_kernel) is two products with S and its update.  As above no factor is a
// quotient of decays.  The first launch computes in 64 bits and rounds what it leaves: sixteen tokens' substitution and
// the terms that cancel between G q and P u cost more than four tokens' do, and in 32 bits the outputs were 1.2 to 1.8 times as
// far from the exact ones as those of the form above (correlated keys the most); so they are at 0.3 to 0.6 of its error (0.4 -
// 1.2e-7 against 0.9 - 2.2e-7), for all that is left in 32 bits is the chain's own sums.  A token's places in W, U, Q and P U
// hang on no later token.
// The chain of the form above is 0.29 us a token of a sequence (2,200 cycles for four tokens, four warps on an
// SM, most of it the latency of shuffles, shared memory and the triangle inside a group); here it is bound by the
// reads of shared memory.  2,048 tokens of 16 heads of 128 x 128: 595 us (500 with one decay a head) there, 316 here; in 32 bits
// throughout it was 295.
constexpr int CC = 16, CS_COLS = 16, CS_THREADS = 256;
constexpr long long CHUNK_SCRATCH = 1ll << 25;      // floats of DeltaWork at most (128 MB): a step of more chunks goes window by window
struct DeltaWork {             // what the first launch leaves of the window's chunks, sixteen rows each, a row a (token, value head)
    float *w, *q, *kd;         // [16 chunks, H, NP]; w and q in the order chunk_place
    float *u, *pu;             // [16 chunks, H, dv]
    float* all;                // [chunk, H, NP]: a chunk's decay of a channel
    int first, chunks;         // the window: numbers of chunks
};
// where channel c lies in a row of w and q: a thread's four channels c, c + 16, c + 32, c + 48 are one 16-byte unit
__device__ __forceinline__ int chunk_place(int c) { return (c & ~63) + (c & 15) * 4 + ((c >> 4) & 3); }
// number of the chunk that starts at token `tok` (counted in the step) of sequence s: different for all chunks of a step
__device__ __forceinline__ int chunk_number(int tok, int s) { return tok / CC + s; }
__device__ __forceinline__ double shfl_xor(double v, int lanes) { return __shfl_xor_sync(0xffffffffu, v, lanes); }

template <int NP, bool CH>
__global__ void __launch_bounds__(256, 2)
delta_chunk_kernel(const DeltaSeq p, const DeltaWork wk, int num_seqs) {
    constexpr int PK = NP + 4;
    __shared__ __align__(16) float sk[CC][PK], sq[CC][PK], sg[CH ? CC : 1][PK];
    __shared__ __align__(16) double s_l[CC][CC], s_p[CC][CC];      // L, P; both 0 where j is later
    __shared__ double s_beta[CC], s_lg[CC], s_eb[CC], s_er[CC];
    __shared__ int s_seq;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, at_chunk = blockIdx.x, number = wk.first + at_chunk, h = blockIdx.y;
    if (tid == 0) s_seq = -1;
    pdl_sync();
    __syncthreads();
    for (int s = tid; s < num_seqs; s += blockDim.x) {
        const int a = p.cu_seqlens[s], n = p.cu_seqlens[s + 1] - a, first = chunk_number(a, s);
        if (n > 0 && number >= first && number < first + (n + CC - 1) / CC) s_seq = s;
    }
    __syncthreads();
    const int s = s_seq;
    if (s < 0) return;
    const int a0 = p.cu_seqlens[s], tok = a0 + (number - chunk_number(a0, s)) * CC, cnt = min(CC, p.cu_seqlens[s + 1] - tok);
    const int d = p.d, dv = p.dv, g = h / (p.H / p.G), channels = 2 * p.G * d + p.H * dv;
    const float* base = p.qkv + (size_t)tok * channels;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
    for (int e = tid; e < CC * (NP / 4); e += 256) {
        const int i = e / (NP / 4), c = (e % (NP / 4)) * 4;
        const bool on = i < cnt && c < d;
        *reinterpret_cast<float4*>(&sk[i][c]) = on ? *reinterpret_cast<const float4*>(base + (size_t)i * channels + (p.G + g) * d + c) : zero;
        *reinterpret_cast<float4*>(&sq[i][c]) = on ? *reinterpret_cast<const float4*>(base + (size_t)i * channels + g * d + c) : zero;
        if (CH) *reinterpret_cast<float4*>(&sg[i][c]) = on ? *reinterpret_cast<const float4*>(p.decay + ((size_t)(tok + i) * p.H + h) * d + c) : one;
    }
    if (tid < CC) {
        s_beta[tid] = tid < cnt ? p.step[(size_t)(tok + tid) * 2 * p.H + h] : 0.f;
        s_lg[tid] = !CH && tid < cnt ? p.step[(size_t)(tok + tid) * 2 * p.H + p.H + h] : 0.f;
    }
    __syncthreads();
    if (!CH && tid < 2 * CC) {         // every exponent is a sum of logarithms, never a difference
        const int i = tid & (CC - 1);
        double x = 0.;
        if (tid < CC)
            for (int e = 0; e <= i; e++) x += s_lg[e];
        else
            for (int e = i + 1; e < CC; e++) x += s_lg[e];
        (tid < CC ? s_eb : s_er)[i] = exp(x);
    }
    // pair sums: a warp takes the pairs of tokens j = warp and 15 - warp with every later one; the thirty-two sums over the
    // warp cost 31 shuffles, and lane l ends with number l: [0 ... 15] k_i . k_j, [16 ... 31] q_i . k_j, i = l & 15
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        const int j = half ? CC - 1 - warp : warp;
        const int e = lane * 4;
        double since[4];               // k_j times the decays after j
        {
            const float4 kj = e < NP ? *reinterpret_cast<const float4*>(&sk[j][e]) : zero;
            since[0] = kj.x, since[1] = kj.y, since[2] = kj.z, since[3] = kj.w;
        }
        double v32[32];
#pragma unroll
        for (int i = 0; i < CC; i++) {
            v32[i] = v32[CC + i] = 0.;
            if (i >= j && e < NP) {
                if (CH && i > j) {
                    const float4 gi = *reinterpret_cast<const float4*>(&sg[CH ? i : 0][e]);
                    since[0] *= gi.x, since[1] *= gi.y, since[2] *= gi.z, since[3] *= gi.w;
                }
                const float4 ki = *reinterpret_cast<const float4*>(&sk[i][e]), qi = *reinterpret_cast<const float4*>(&sq[i][e]);
                v32[i] = fma((double)ki.x, since[0], fma((double)ki.y, since[1], fma((double)ki.z, since[2], ki.w * since[3])));
                v32[CC + i] = fma((double)qi.x, since[0], fma((double)qi.y, since[1], fma((double)qi.z, since[2], qi.w * since[3])));
            }
        }
#pragma unroll
        for (int n = 16; n >= 1; n >>= 1) {
            const bool up = (lane & n) != 0;
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (i < n) v32[i] = (up ? v32[n + i] : v32[i]) + shfl_xor(up ? v32[i] : v32[n + i], n);
        }
        double dot = v32[0];
        const int i = lane & 15;
        if (!CH) {
            double between = 0.;       // the decays' logarithms after j up to i, added up and not subtracted
            for (int l = j + 1; l <= i; l++) between += s_lg[l];
            dot *= exp(between);
        }
        if (lane < 16)
            s_l[i][j] = i > j ? s_beta[i] * dot : 0.;
        else
            s_p[i][j] = i >= j ? dot : 0.;
    }
    __syncthreads();
    double x[CC];
    auto solve = [&]() {               // x <- (I + L)^-1 x
#pragma unroll
        for (int i = 1; i < CC; i++) {
            asm volatile("" ::: "memory");       // (or all of L is fetched first)
#pragma unroll
            for (int j = 0; j < i; j += 2) {
                const double2 l2 = *reinterpret_cast<const double2*>(&s_l[i][j]);
                x[i] = fma(-l2.x, x[j], x[i]);
                if (j + 1 < i) x[i] = fma(-l2.y, x[j + 1], x[i]);
            }
        }
    };
    auto pair_sum = [&](int i) {       // (P x)_i
        double r = 0.;
#pragma unroll
        for (int j = 0; j < CC; j += 2)
            if (j <= i) {
                const double2 p2 = *reinterpret_cast<const double2*>(&s_p[i][j]);
                r = fma(p2.x, x[j], r);
                if (j + 1 <= i) r = fma(p2.y, x[j + 1], r);
            }
        return r;
    };
    if (tid < NP) {
        const int c = tid, at = chunk_place(c);
        const size_t row = ((size_t)at_chunk * CC * p.H + h) * NP, pitch = (size_t)p.H * NP;
        double all = 1.;
#pragma unroll
        for (int i = 0; i < CC; i++) {
            if (CH) all *= sg[CH ? i : 0][c]; else all = s_eb[i];
            x[i] = s_beta[i] * (sk[i][c] * all);
        }
        wk.all[((size_t)at_chunk * p.H + h) * NP + c] = (float)all;
        double since = 1.;
#pragma unroll
        for (int i = CC - 1; i >= 0; i--) {
            if (i < cnt) wk.kd[row + i * pitch + c] = (float)(sk[i][c] * (CH ? since : s_er[i]));
            if (CH) since *= sg[CH ? i : 0][c];
        }
        solve();
        all = 1.;
#pragma unroll
        for (int i = 0; i < CC; i++) {
            asm volatile("" ::: "memory");
            if (CH) all *= sg[CH ? i : 0][c]; else all = s_eb[i];
            const double q = sq[i][c] * all - pair_sum(i);
            if (i < cnt) wk.w[row + i * pitch + at] = (float)x[i], wk.q[row + i * pitch + at] = (float)q;
        }
    } else {
        for (int c = tid - NP; c < dv; c += 256 - NP) {
            const float* v = base + 2 * p.G * d + (size_t)h * dv + c;
#pragma unroll
            for (int i = 0; i < CC; i++) x[i] = i < cnt ? s_beta[i] * v[(size_t)i * channels] : 0.;
            solve();
            const size_t row = ((size_t)at_chunk * CC * p.H + h) * dv + c, pitch = (size_t)p.H * dv;
#pragma unroll
            for (int i = 0; i < CC; i++) {
                asm volatile("" ::: "memory");
                const double r = pair_sum(i);
                if (i < cnt) wk.u[row + i * pitch] = (float)x[i], wk.pu[row + i * pitch] = (float)r;
            }
        }
    }
}

// grid (ceil(dv / 16), heads, sequences): a block carries 16 columns of S in shared memory through its sequence's chunks in the
// window.
// A thread of the first product holds 8 of the 32 rows [W; Q] x 4 columns over every 16th channel (the sum over
// the 16 threads that share them is 30 shuffles) and ends with two elements of u or two outputs; then half of the threads
// update the state, 4 channels x 4 columns each.
template <int NP>
struct ChunkSmem {
    static constexpr int STAGE = 3 * CC * NP + 2 * CC * CS_COLS + NP;      // W | Q | D k | U | P U | decays
    static constexpr int SPITCH = CS_COLS + 4;
    static constexpr int FLOATS = 2 * STAGE + NP * SPITCH + CC * SPITCH;
};
template <int NP>
__global__ void __launch_bounds__(CS_THREADS, 2)
delta_chunk_scan_kernel(const DeltaSeq p, const DeltaWork wk, float* __restrict__ o) {
    using L = ChunkSmem<NP>;
    constexpr int SP = L::SPITCH;
    extern __shared__ __align__(16) float sm[];
    float* sS = sm + 2 * L::STAGE;     // [NP][SP]
    float* sU = sS + NP * SP;          // [16][SP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.y, s = blockIdx.z, c0 = blockIdx.x * CS_COLS, d = p.d, dv = p.dv;
    pdl_sync();
    const int tok0 = p.cu_seqlens[s], cnt = p.cu_seqlens[s + 1] - tok0;
    const int number0 = chunk_number(tok0, s);        // (counted from the window's first chunk the sequence's first is number0 - first)
    const int begin = max(0, wk.first - number0) * CC, end = min(cnt, (wk.first + wk.chunks - number0) * CC);
    if (begin >= end) return;
    float* S = p.state + (size_t)p.slots[s] * p.state_pitch + (size_t)h * d * dv;
    const int ncols = min(CS_COLS, dv - c0);
    auto stage = [&](int t0, int buf) {
        float* dst = sm + buf * L::STAGE;
        const size_t at_chunk = number0 - wk.first + t0 / CC, row0 = at_chunk * CC * p.H + h;
        for (int e = tid; e < 3 * CC * (NP / 4); e += CS_THREADS) {
            const int which = e / (CC * (NP / 4)), i = e / (NP / 4) % CC, c = (e % (NP / 4)) * 4;
            const bool on = t0 + i < cnt;
            const float* src = which == 0 ? wk.w : which == 1 ? wk.q : wk.kd;
            cp_zfill(dst + which * CC * NP + i * NP + c, on ? src + (row0 + (size_t)i * p.H) * NP + c : src, 16, on);
        }
        float* du = dst + 3 * CC * NP;
        if (tid < 128) {
            const int i = (tid & 63) >> 2, c = (tid & 3) * 4, which = tid >> 6;
            const bool on = t0 + i < cnt && c < ncols;
            const float* src = which ? wk.pu : wk.u;
            cp_zfill(du + which * CC * CS_COLS + i * CS_COLS + c, on ? src + (row0 + (size_t)i * p.H) * dv + c0 + c : src, 16, on);
        } else if (tid < 128 + NP / 4) {
            const int c = (tid - 128) * 4;
            cp_zfill(du + 2 * CC * CS_COLS + c, wk.all + (at_chunk * p.H + h) * NP + c, 16, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(begin, 0);
    for (int e = tid; e < NP * CS_COLS; e += CS_THREADS) {
        const int r = e / CS_COLS, c = e % CS_COLS;
        sS[r * SP + c] = r < d && c < ncols ? S[(size_t)r * dv + c0 + c] : 0.f;
    }
    const int ks = lane & 15, cg = ((warp & 1) * 2 + (lane >> 4)) * 4, tg = warp >> 1;
    for (int t0 = begin, buf = 0; t0 < end; t0 += CC, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                               // the chunk is there, the state and the other buffer are at rest
        if (t0 + CC < end) stage(t0 + CC, buf ^ 1);
        const float* st = sm + buf * L::STAGE;
        const float* du = st + 3 * CC * NP;
        {
            float acc[32];
#pragma unroll
            for (int i = 0; i < 32; i++) acc[i] = 0.f;
            const float* rows = st + tg * 8 * NP + ks * 4;
#pragma unroll
            for (int it = 0; it < NP / 64; it++) {
                float4 sv[4];
#pragma unroll
                for (int r = 0; r < 4; r++) sv[r] = *reinterpret_cast<const float4*>(sS + (it * 64 + r * 16 + ks) * SP + cg);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float4 w4 = *reinterpret_cast<const float4*>(rows + i * NP + it * 64);
                    const float wr[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        acc[4 * i] = fmaf(wr[r], sv[r].x, acc[4 * i]), acc[4 * i + 1] = fmaf(wr[r], sv[r].y, acc[4 * i + 1]);
                        acc[4 * i + 2] = fmaf(wr[r], sv[r].z, acc[4 * i + 2]), acc[4 * i + 3] = fmaf(wr[r], sv[r].w, acc[4 * i + 3]);
                    }
                }
            }
            // thirty-two sums over sixteen lanes: a lane ends with two neighbouring ones
            float v16[16], v8[8], v4[4], v2[2];
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const bool up = (lane & 8) != 0;
                v16[i] = (up ? acc[16 + i] : acc[i]) + __shfl_xor_sync(0xffffffffu, up ? acc[i] : acc[16 + i], 8);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const bool up = (lane & 4) != 0;
                v8[i] = (up ? v16[8 + i] : v16[i]) + __shfl_xor_sync(0xffffffffu, up ? v16[i] : v16[8 + i], 4);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const bool up = (lane & 2) != 0;
                v4[i] = (up ? v8[4 + i] : v8[i]) + __shfl_xor_sync(0xffffffffu, up ? v8[i] : v8[4 + i], 2);
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const bool up = (lane & 1) != 0;
                v2[i] = (up ? v4[2 + i] : v4[i]) + __shfl_xor_sync(0xffffffffu, up ? v4[i] : v4[2 + i], 1);
            }
            // rows of W: two elements of u; rows of Q: two outputs (dv is a multiple of four)
            const int i = (tg & 1) * 8 + (ks >> 1), c = cg + (ks & 1) * 2;
            const float2 more = *reinterpret_cast<const float2*>(du + (tg >> 1) * CC * CS_COLS + i * CS_COLS + c);
            if (tg < 2)
                *reinterpret_cast<float2*>(sU + i * SP + c) = make_float2(more.x - v2[0], more.y - v2[1]);
            else if (t0 + i < cnt && c < ncols) {
                float* out = o + ((size_t)(tok0 + t0 + i) * p.H + h) * dv + c0 + c;
                out[0] = v2[0] + more.x, out[1] = v2[1] + more.y;
            }
        }
        __syncthreads();
        if (tid < CS_THREADS / 2) {
            // the state: four neighbouring channels x four columns a thread (of half of the threads: the reads of shared memory are what it
            // takes, and 2 x 4 of all of them need twice as many: 2,048 tokens 223 / 245 us); what the chunk adds is summed by itself, so that the
            // state is rounded once a chunk
            for (int r0 = (tid >> 2) * 4; r0 < NP; r0 += CS_THREADS / 2) {
                const int cc = (tid & 3) * 4;
                float4 a[4];
#pragma unroll
                for (int r = 0; r < 4; r++) a[r] = make_float4(0.f, 0.f, 0.f, 0.f);
                const float* kd = st + 2 * CC * NP + r0;
#pragma unroll
                for (int j = 0; j < CC; j++) {
                    const float4 k4 = *reinterpret_cast<const float4*>(kd + j * NP), u4 = *reinterpret_cast<const float4*>(sU + j * SP + cc);
                    const float k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        a[r].x = fmaf(k[r], u4.x, a[r].x), a[r].y = fmaf(k[r], u4.y, a[r].y);
                        a[r].z = fmaf(k[r], u4.z, a[r].z), a[r].w = fmaf(k[r], u4.w, a[r].w);
                    }
                }
                const float4 al = *reinterpret_cast<const float4*>(du + 2 * CC * CS_COLS + r0);
                const float all[4] = {al.x, al.y, al.z, al.w};
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    float4* at = reinterpret_cast<float4*>(sS + (r0 + r) * SP + cc);
                    const float4 before = *at;
                    *at = make_float4(fmaf(all[r], before.x, a[r].x), fmaf(all[r], before.y, a[r].y), fmaf(all[r], before.z, a[r].z),
                                      fmaf(all[r], before.w, a[r].w));
                }
            }
        }
    }
    __syncthreads();
    for (int e = tid; e < NP * CS_COLS; e += CS_THREADS) {
        const int r = e / CS_COLS, c = e % CS_COLS;
        if (r < d && c < ncols) S[(size_t)r * dv + c0 + c] = sS[r * SP + c];
    }
}

bool aligned16(const void* p) { return (uintptr_t)p % 16 == 0; }

// Chunk numbers of a step, and floats that the first launch leaves of one chunk.
long long chunk_numbers(long long T, int num_seqs) { return T / CC + num_seqs + 1; }
long long chunk_floats(int H, int d, int dv) {
    const long long NP = d <= 64 ? 64 : 128;
    return H * (CC * (3 * NP + 2ll * dv) + NP);
}
// Chunks of a window: all of the step's if their results find room, as many as do otherwise.
long long chunk_window(long long T, int num_seqs, int H, int d, int dv) {
    const long long n = chunk_numbers(T, num_seqs), room = CHUNK_SCRATCH / chunk_floats(H, d, dv);
    return n < room ? n : room;
}

}  // namespace

// proj: [T, ld] 32-bit: q (G * d columns), k (G * d), v (H * dv), b and a (a column a value head) from b_at and
// a_at; taps_w: [taps, channels]; state: (taps - 1) * channels floats a slot from the pointer given; out: [T, channels]
// 32-bit; step: [T, 2 H] 32-bit (beta, then the decay's logarithm).  `shift`: the step brings one token a sequence and the state moves on here.
// With `decay` not null there is a decay a channel: a_rows [T, lda] holds a (H * d columns), dt_bias [H * d], and decay
// [T, H * d] receives the decays (a_at is not read then).
MOE_API int moe_delta_prepare(const float* proj, long long ld, int b_at, int a_at, const float* taps_w, int taps,
                              float* state, long long state_pitch, const float* a_log, const float* dt_bias,
                              const int* seq_of_token, const int* cu_seqlens, const int* slots, int num_tokens, int H,
                              int G, int d, int dv, float eps, float q_scale, int shift, float* out, float* step,
                              const float* a_rows, long long lda, float* decay, cudaStream_t stream) {
    if (num_tokens <= 0) return 0;
    const long long channels = 2LL * G * d + (long long)H * dv;
    if (!proj || !taps_w || !a_log || !dt_bias || !seq_of_token || !cu_seqlens || !slots || !out || !step || H <= 0 || G <= 0 ||
        H % G || d <= 0 || d > DP_MAX_D || dv <= 0 || taps < 1 || taps > 16 || (taps > 1 && !state) || ld < channels ||
        b_at < 0 || b_at + H > ld || (decay ? !a_rows || lda < (long long)H * d : a_at < 0 || a_at + H > ld) || (taps > 1 && state_pitch < (taps - 1) * channels))
        return (int)cudaErrorInvalidValue;
    const DeltaPrep p{proj, ld, b_at, a_at, taps_w, state, state_pitch, a_log, dt_bias, seq_of_token, cu_seqlens, slots,
                      num_tokens, taps, H, G, d, dv, shift, eps, q_scale, out, step, a_rows, lda, decay};
    const bool vec = d % 4 == 0 && dv % 4 == 0 && ld % 4 == 0 && state_pitch % 4 == 0 && aligned16(proj) && aligned16(taps_w) &&
                     aligned16(state) && aligned16(out) &&
                     (!decay || (lda % 4 == 0 && aligned16(a_rows) && aligned16(decay) && aligned16(dt_bias)));
    const int per = vec ? 128 : 32;
    const int items = 2 * G + (H * dv + per - 1) / per + 1 + (decay ? (H * d + per - 1) / per : 0);
    // many tokens: runs of them
    if (vec && !shift && num_tokens >= 128 && d <= 128 && taps >= 2 && taps <= 4) {
        const dim3 runs((num_tokens + DP_RUN - 1) / DP_RUN, (items + DP_WARPS - 1) / DP_WARPS);
        if (runs.y > 65535) return (int)cudaErrorInvalidValue;
        const auto kernel = taps == 2 ? delta_prepare_run_kernel<2> : taps == 3 ? delta_prepare_run_kernel<3> : delta_prepare_run_kernel<4>;
        return launch_pdl(kernel, runs, dim3(DP_WARPS * 32), 0, stream, p);
    }
    // few tokens: a warp an item; many: a block a token
    const dim3 grid(num_tokens, num_tokens >= 128 ? 1 : (items + DP_WARPS - 1) / DP_WARPS);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
#define PREP(W_, T_) return launch_pdl(delta_prepare_kernel<W_, T_>, grid, dim3(DP_WARPS * 32), 0, stream, p)
    if (vec) {
        if (taps == 2) PREP(4, 2);
        if (taps == 3) PREP(4, 3);
        if (taps == 4) PREP(4, 4);
        PREP(4, 0);
    }
    if (taps == 4) PREP(1, 4);
    PREP(1, 0);
#undef PREP
}

// One token a sequence.  qkv, step: as moe_delta_prepare leaves them; state: H * d * dv floats a slot from the pointer
// given; decay: [T, H * d] or null; gate: [T, H * dv] 32-bit logits, rows of ldg, through gate_fn (GATE_*); norm_w: [H * dv]; out: [T, H * dv] in out_dt (rows of no
// sequence become zeros).  Returns -1, with nothing launched, for sizes it does not take.
MOE_API int moe_delta_step(const float* qkv, const float* step, float* state, long long state_pitch, const float* gate,
                           long long ldg, const float* norm_w, float norm_eps, const int* seq_of_token,
                           const int* cu_seqlens, const int* slots, int num_tokens, int num_seqs, int H, int G, int d,
                           int dv, const float* decay, int gate_fn, void* out, int out_dt, cudaStream_t stream) {
    if (num_seqs <= 0 || num_tokens <= 0) return 0;
    if (!qkv || !step || !state || !gate || !norm_w || !seq_of_token || !cu_seqlens || !slots || !out || H <= 0 || G <= 0 ||
        H % G || d <= 0 || dv <= 0 || ldg < (long long)H * dv || state_pitch < (long long)H * d * dv || num_seqs > 65535)
        return (int)cudaErrorInvalidValue;
    if (dv % 4 || dv > 512 || d > 256 || state_pitch % 4 || !aligned16(state)) return -1;
    const int cg = dv / 4, kp = 256 / cg, units = (d + kp - 1) / kp;
    const size_t smem = ((size_t)2 * ((d + 1) / 2 * 2) + dv + (size_t)kp * dv + (decay ? d : 0)) * sizeof(float);
    if (units > 32 || smem > 48 * 1024 || d % 2) return -1;
    const DeltaSeq p{qkv, step, state, state_pitch, cu_seqlens, slots, H, G, d, dv, decay};
#define STEP_C(OT_, U_, C_)                                                                                            \
    return launch_pdl(delta_step_kernel<OT_, U_, C_>, dim3(H, num_seqs), dim3(256), smem, stream, p, gate, ldg, norm_w, norm_eps, \
                      seq_of_token, num_tokens, gate_fn, (OT_*)out)
#define STEP(OT_, U_)                                                                                                  \
    do {                                                                                                               \
        if (decay) STEP_C(OT_, U_, true);                                                                              \
        STEP_C(OT_, U_, false);                                                                                        \
    } while (0)
#define STEP_U(OT_)                                                                                                    \
    do {                                                                                                               \
        if (units <= 4) STEP(OT_, 4);                                                                                  \
        if (units <= 8) STEP(OT_, 8);                                                                                  \
        if (units <= 16) STEP(OT_, 16);                                                                                \
        STEP(OT_, 32);                                                                                                 \
    } while (0)
    if (out_dt == DT_F32) STEP_U(float);
    STEP_U(__nv_bfloat16);
#undef STEP_U
#undef STEP
#undef STEP_C
}

// SMs of the current device.
MOE_API int moe_scan_sms() { return scan_sms(); }

// Floats of scratch with which moe_delta_scan takes the form over chunks of sixteen tokens; 0: it takes the other one.
MOE_API long long moe_delta_chunk_floats(long long num_tokens, int num_seqs, int H, int G, int d, int dv) {
    if (num_tokens <= 0 || num_seqs <= 0 || d <= 0 || d > 128 || d % 4 || dv <= 0 || dv % 4 || H <= 0 || H > 65535 || num_seqs > 65535) return 0;
    return chunk_window(num_tokens, num_seqs, H, d, dv) * chunk_floats(H, d, dv);
}

// Several tokens a sequence; o: [T, H * dv] 32-bit (rows of no sequence are left alone).  `work`: moe_delta_chunk_floats
// floats, or null for the form of four tokens at a time.
MOE_API int moe_delta_scan(const float* qkv, const float* step, float* state, long long state_pitch, const int* cu_seqlens,
                           const int* slots, int num_tokens, int num_seqs, int H, int G, int d, int dv, const float* decay,
                           float* o, float* work, cudaStream_t stream) {
    if (num_seqs <= 0) return 0;
    if (!qkv || !step || !state || !cu_seqlens || !slots || !o || H <= 0 || G <= 0 || H % G || d <= 0 || d > 256 || dv <= 0 ||
        state_pitch < (long long)H * d * dv || H > 65535 || num_seqs > 65535)
        return (int)cudaErrorInvalidValue;
    const DeltaSeq p{qkv, step, state, state_pitch, cu_seqlens, slots, H, G, d, dv, decay};
    if (work && moe_delta_chunk_floats(num_tokens, num_seqs, H, G, d, dv) > 0 && aligned16(qkv) && aligned16(decay) && aligned16(work)) {
        const int NP = d <= 64 ? 64 : 128;
        DeltaWork wk;
        const long long numbers = chunk_numbers(num_tokens, num_seqs), window = chunk_window(num_tokens, num_seqs, H, d, dv);
        const size_t rows = (size_t)window * CC * H;
        wk.w = work, wk.q = wk.w + rows * NP, wk.kd = wk.q + rows * NP, wk.u = wk.kd + rows * NP, wk.pu = wk.u + rows * dv;
        wk.all = wk.pu + rows * dv;
        const dim3 chain((dv + CS_COLS - 1) / CS_COLS, H, num_seqs);
#define CHUNK(NP_, C_)                                                                                                  \
    do {                                                                                                               \
        const size_t smem = scan_smem(ChunkSmem<NP_>::FLOATS * sizeof(float), (long long)chain.x * chain.y * chain.z); \
        cudaError_t e = cudaFuncSetAttribute(delta_chunk_scan_kernel<NP_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        if (e != cudaSuccess) return (int)e;                                                                           \
        for (long long at = 0; at < numbers; at += window) {                                                           \
            wk.first = (int)at, wk.chunks = (int)(numbers - at < window ? numbers - at : window);                      \
            int rc = launch_pdl(delta_chunk_kernel<NP_, C_>, dim3(wk.chunks, H), dim3(256), 0, stream, p, wk, num_seqs); \
            if (rc) return rc;                                                                                         \
            delta_chunk_scan_kernel<NP_><<<chain, CS_THREADS, smem, stream>>>(p, wk, o);                               \
            if ((rc = launch_status())) return rc;                                                                     \
        }                                                                                                              \
        return 0;                                                                                                      \
    } while (0)
        if (NP == 64) {
            if (decay) CHUNK(64, true);
            CHUNK(64, false);
        }
        if (decay) CHUNK(128, true);
        CHUNK(128, false);
#undef CHUNK
    }
    // few blocks: the narrow form puts twice as many on the SMs
    const bool narrow = d > 64 && (long long)((dv + dcols(16) - 1) / dcols(16)) * H * num_seqs * 2 <= scan_sms();
    const int cols = dcols(narrow ? 32 : 16);
    const dim3 grid((dv + cols - 1) / cols, H, num_seqs);
    const bool vec = d % 4 == 0 && dv % 4 == 0 && aligned16(qkv) && aligned16(decay);
    // An ordinary launch: blocks that are placed while the kernel before still occupies some SMs end up several to
    // an SM beside empty ones, and a scan is as slow as its most crowded SM.
#define SCAN_V(RPT_, KP_, V_, C_)                                                                                      \
    do {                                                                                                               \
        const size_t smem = scan_smem(delta_scan_floats<RPT_, KP_, C_>() * sizeof(float), (long long)grid.x * grid.y * grid.z); \
        if (smem > 48 * 1024) {                                                                                        \
            cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel<RPT_, KP_, V_, C_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            if (e != cudaSuccess) return (int)e;                                                                       \
        }                                                                                                              \
        delta_scan_kernel<RPT_, KP_, V_, C_><<<grid, DTHREADS, smem, stream>>>(p, o);                                  \
        return launch_status();                                                                                        \
    } while (0)
#define SCAN(RPT_, KP_)                                                                                                \
    do {                                                                                                               \
        if (decay) {                                                                                                   \
            if (vec) SCAN_V(RPT_, KP_, true, true);                                                                    \
            SCAN_V(RPT_, KP_, false, true);                                                                            \
        }                                                                                                              \
        if (vec) SCAN_V(RPT_, KP_, true, false);                                                                       \
        SCAN_V(RPT_, KP_, false, false);                                                                               \
    } while (0)
    if (d <= 64) SCAN(4, 16);
    if (narrow) {
        if (d <= 128) SCAN(4, 32);
        SCAN(8, 32);
    }
    if (d <= 128) SCAN(8, 16);
    SCAN(16, 16);
#undef SCAN
#undef SCAN_V
}
