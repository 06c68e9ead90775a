// Kernels of the gated delta rule mixer with one decay per head and key channel.
//
// A request's state slot holds, in 32-bit floats: per head the matrix S (dim x vdim), stored
// column by column ([heads][vdim][dim]), then the last taps - 1 inputs of the short convolutions
// ([taps - 1][channels], oldest first).
//
//  * delta_prep (delta_prep_tile: sixteen tokens at a time): per token the short causal convolution (per channel, over the step's earlier
//    tokens of the same request and, before them, the slot's kept inputs) and silu of q, k, v;
//    q and k as unit vectors per head (q also times dim^-1/2); beta = sigmoid(.); the decay
//    g = exp(-exp(A_log[head]) * softplus(a + dt_bias)).
//  * delta_conv_tail: the slot's kept inputs moved on by the step's tokens.
//  * delta_rule: per token, in order:  S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;
//    o = S^T q.  Columns of S do not interact: a block owns some columns of one head of one
//    request, a group of TPC lanes one column (lane j of the group holds rows R j .. R j + R - 1),
//    and walks the request's tokens of this step in order, eight at a time through shared memory.
//    Each sum over rows is taken in an order that depends on `dim` alone.
//  * gated_rms_heads: o / rms(o) per head, times a weight, times sigmoid(gate).
// Everything here is 32-bit.
#include "gated_rows.cuh"
#include <math.h>

namespace {

__device__ __forceinline__ float silu_f(float y) { return y / (1.0f + expf(-y)); }
__device__ __forceinline__ float sigmoid_f(float y) { return 1.0f / (1.0f + expf(-y)); }
__device__ __forceinline__ float softplus_f(float y) { return y > 20.0f ? y : log1pf(expf(y)); }

// grid: (tokens, units).  The units of a token: the q heads, the k heads (convolution, silu, unit
// norm over `dim` channels each), the v heads (convolution and silu over `vdim` channels each), the
// heads' decays (`dim` values each), and one unit for the betas.  channels = 2 * kv_heads * dim +
// heads * vdim; qkvb rows hold the channels and then `heads` betas.
__device__ __forceinline__ void
delta_prep_unit(int n, int unit, float* y, float* red,
                const float* __restrict__ qkvb, int ld, const float* __restrict__ a,
                  const float* __restrict__ conv_w, const float* __restrict__ A_log,
                  const float* __restrict__ dt_bias, const float* __restrict__ state, long long state_stride,
                  const int* __restrict__ slots, const int* __restrict__ seq_of_token,
                  const int* __restrict__ cu_q, float* __restrict__ q_out, float* __restrict__ k_out,
                  float* __restrict__ v_out, float* __restrict__ beta, float* __restrict__ decay,
                  int heads, int kv_heads, int dim, int vdim, int taps, int num_slots, int* err) {
    int tid = threadIdx.x;
    int qk = kv_heads * dim, channels = 2 * qk + heads * vdim;
    if (unit == 2 * kv_heads + 2 * heads) {  // the betas
        for (int h = tid; h < heads; h += blockDim.x) beta[(size_t)n * heads + h] = sigmoid_f(qkvb[(size_t)n * ld + channels + h]);
        return;
    }
    if (unit >= 2 * kv_heads + heads) {  // a head's decays
        int h = unit - 2 * kv_heads - heads;
        float rate = expf(A_log[h]);
        for (int d = tid; d < dim; d += blockDim.x) {
            size_t i = (size_t)n * heads * dim + h * dim + d;
            decay[i] = expf(-rate * softplus_f(a[i] + dt_bias[h * dim + d]));
        }
        return;
    }
    int seq = seq_of_token[n];
    int t = n - cu_q[seq];  // the token's place among the request's tokens of this step
    int slot = slots[seq];
    if (slot < 0 || slot >= num_slots) {
        if (tid == 0) ie_report(err, IE_ERR_PAGE, slot, n);
        return;
    }
    bool is_v = unit >= 2 * kv_heads;
    int width = is_v ? vdim : dim;
    int first = is_v ? 2 * qk + (unit - 2 * kv_heads) * vdim : unit * dim;  // the unit's first channel
    const float* tail = state + (size_t)slot * state_stride + (size_t)heads * dim * vdim;
    float ss = 0.f;
    for (int i = tid; i < width; i += blockDim.x) {
        int c = first + i;
        float acc = 0.f;
        for (int j = 0; j < taps; ++j) {
            int back = taps - 1 - j;  // this tap looks `back` tokens back
            float x = (t - back >= 0) ? qkvb[(size_t)(n - back) * ld + c]
                                      : tail[(size_t)(taps - 1 + t - back) * channels + c];
            acc = fmaf(conv_w[(size_t)c * taps + j], x, acc);
        }
        float sv = silu_f(acc);
        if (is_v) v_out[(size_t)n * heads * vdim + (c - 2 * qk)] = sv;
        else { y[i] = sv; ss = fmaf(sv, sv, ss); }
    }
    if (is_v) return;
    ss = warp_sum(ss);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    float f = 1.0f / sqrtf(((red[0] + red[1]) + (red[2] + red[3])) + 1e-6f);
    bool is_q = unit < kv_heads;
    if (is_q) f *= 1.0f / sqrtf((float)dim);
    float* dst = (is_q ? q_out : k_out) + (size_t)n * qk + (is_q ? unit : unit - kv_heads) * dim;
    for (int i = tid; i < dim; i += blockDim.x) dst[i] = y[i] * f;
    __syncthreads();  // (y and red are used again by the block's next unit)
}

// grid: (tokens, blocks per token); a block takes the token's units blockIdx.y, blockIdx.y + gridDim.y, ...
// (a block per unit when the step has few tokens, a few blocks per token when it has many).
__global__ void __launch_bounds__(128)
delta_prep_kernel(const float* __restrict__ qkvb, int ld, const float* __restrict__ a,
                  const float* __restrict__ conv_w, const float* __restrict__ A_log,
                  const float* __restrict__ dt_bias, const float* __restrict__ state, long long state_stride,
                  const int* __restrict__ slots, const int* __restrict__ seq_of_token,
                  const int* __restrict__ cu_q, float* __restrict__ q_out, float* __restrict__ k_out,
                  float* __restrict__ v_out, float* __restrict__ beta, float* __restrict__ decay,
                  int heads, int kv_heads, int dim, int vdim, int taps, int num_slots, int* err) {
    extern __shared__ float y[];  // [max(dim, vdim)]: one unit's channels after the convolution
    __shared__ float red[4];
    ie_pdl_trigger();
    ie_pdl_wait();
    int units = 2 * kv_heads + 2 * heads + 1;
    for (int unit = blockIdx.y; unit < units; unit += gridDim.y)
        delta_prep_unit(blockIdx.x, unit, y, red, qkvb, ld, a, conv_w, A_log, dt_bias, state, state_stride, slots,
                        seq_of_token, cu_q, q_out, k_out, v_out, beta, decay, heads, kv_heads, dim, vdim, taps,
                        num_slots, err);
}

// The same for many tokens.  grid: (blocks of PT_TOKENS tokens, units); a thread takes a channel of the unit through its block's
// tokens, so an input is read once and not once per tap, and sixteen loads are on their way at once (2,048 tokens of 16 heads of
// 128 x 128: 147 us a token at a time, bound by the units' chains of loads and barriers; 102 with three blocks an SM, whose 168
// registers a thread left too few loads in flight; 63 with five, 57 since the
// block's rows are asked for before it is known whose they are).  q and k: `dim` at most 128, one
// channel per thread, whose squares sixteen tokens add up together (every exchange halves the sums a lane still holds).
constexpr int PT_TOKENS = 16;
template <int TAPS>
__global__ void __launch_bounds__(128, 5)
delta_prep_tile_kernel(const float* __restrict__ qkvb, int ld, const float* __restrict__ a,
                       const float* __restrict__ conv_w, const float* __restrict__ A_log,
                       const float* __restrict__ dt_bias, const float* __restrict__ state, long long state_stride,
                       const int* __restrict__ slots, const int* __restrict__ seq_of_token,
                       const int* __restrict__ cu_q, float* __restrict__ q_out, float* __restrict__ k_out,
                       float* __restrict__ v_out, float* __restrict__ beta, float* __restrict__ decay, int num_tokens,
                       int heads, int kv_heads, int dim, int vdim, int num_slots, int* err) {
    __shared__ float red[4][PT_TOKENS];
    ie_pdl_trigger();
    ie_pdl_wait();
    const int n0 = blockIdx.x * PT_TOKENS, cnt = min(PT_TOKENS, num_tokens - n0), unit = blockIdx.y, tid = threadIdx.x;
    const int qk = kv_heads * dim, channels = 2 * qk + heads * vdim;
    if (unit == 2 * kv_heads + 2 * heads) {  // the betas
        for (int i = tid; i < cnt * heads; i += 128) {
            const size_t n = (size_t)(n0 + i / heads);
            beta[n * heads + i % heads] = sigmoid_f(qkvb[n * ld + channels + i % heads]);
        }
        return;
    }
    if (unit >= 2 * kv_heads + heads) {  // a head's decays
        const int h = unit - 2 * kv_heads - heads;
        const float rate = expf(A_log[h]);
        for (int d = tid; d < dim; d += 128) {
            const float bias = dt_bias[h * dim + d];
            const size_t at = (size_t)n0 * heads * dim + h * dim + d, step = (size_t)heads * dim;
            float v[PT_TOKENS];
#pragma unroll
            for (int i = 0; i < PT_TOKENS; ++i) v[i] = i < cnt ? a[at + i * step] : 0.f;
#pragma unroll
            for (int i = 0; i < PT_TOKENS; ++i)
                if (i < cnt) decay[at + i * step] = expf(-rate * softplus_f(v[i] + bias));
        }
        return;
    }
    const bool is_v = unit >= 2 * kv_heads;
    const int width = is_v ? vdim : dim;
    const int first_channel = is_v ? 2 * qk + (unit - 2 * kv_heads) * vdim : unit * dim;
    const size_t tail_at = (size_t)heads * dim * vdim;
    for (int c0 = 0; c0 < width; c0 += 128) {  // (q and k: once)
        const int i0 = c0 + tid, c = first_channel + i0;
        const bool live = i0 < width;
        float y[PT_TOKENS], w[TAPS];
#pragma unroll
        for (int j = 0; j < TAPS; ++j) w[j] = live ? conv_w[(size_t)c * TAPS + j] : 0.f;
        // The rows of the block and those before it, on their way before it is known which request's they are.
        const int seq0 = seq_of_token[n0];
        float in[PT_TOKENS + TAPS - 1];
        if (cnt == PT_TOKENS) {
            const float* row = qkvb + (size_t)n0 * ld + c;
#pragma unroll
            for (int i = 0; i < PT_TOKENS + TAPS - 1; ++i) {
                const int at = i - (TAPS - 1);  // (negative: that many rows before the block)
                in[i] = live && n0 + at >= 0 ? row[(ptrdiff_t)at * ld] : 0.f;
            }
        }
        const int start = cu_q[seq0], end = cu_q[seq0 + 1], slot = slots[seq0];
        if (cnt == PT_TOKENS && n0 + PT_TOKENS <= end) {  // (all of one request)
            const int t0 = n0 - start;
            if (slot < 0 || slot >= num_slots) {
                if (tid == 0) ie_report(err, IE_ERR_PAGE, slot, n0);
                return;
            }
            if (live && t0 < TAPS - 1) {  // the first are the kept ones
                const float* tail = state + (size_t)slot * state_stride + tail_at;
#pragma unroll
                for (int i = 0; i < TAPS - 1; ++i)
                    if (i + t0 < TAPS - 1) in[i] = tail[(size_t)(i + t0) * channels + c];
            }
#pragma unroll
            for (int i = 0; i < PT_TOKENS; ++i) {
                float acc = 0.f;
#pragma unroll
                for (int j = 0; j < TAPS; ++j) acc = fmaf(w[j], in[i + j], acc);
                y[i] = silu_f(acc);
            }
        } else {
#pragma unroll
            for (int i = 0; i < PT_TOKENS; ++i) {
                y[i] = 0.f;
                if (i < cnt) {
                    const int n = n0 + i, seq = seq_of_token[n], t = n - cu_q[seq], slot = slots[seq];
                    if (slot < 0 || slot >= num_slots) {
                        if (tid == 0) ie_report(err, IE_ERR_PAGE, slot, n);
                    } else if (live) {
                        const float* tail = state + (size_t)slot * state_stride + tail_at;
                        float acc = 0.f;
#pragma unroll
                        for (int j = 0; j < TAPS; ++j) {
                            const int back = TAPS - 1 - j;
                            acc = fmaf(w[j], t - back >= 0 ? qkvb[(size_t)(n - back) * ld + c] : tail[(size_t)(TAPS - 1 + t - back) * channels + c], acc);
                        }
                        y[i] = silu_f(acc);
                    }
                }
            }
        }
        if (is_v) {
            if (live)
#pragma unroll
                for (int i = 0; i < PT_TOKENS; ++i)
                    if (i < cnt) v_out[(size_t)(n0 + i) * heads * vdim + (c - 2 * qk)] = y[i];
            continue;
        }
        float part[PT_TOKENS];
#pragma unroll
        for (int i = 0; i < PT_TOKENS; ++i) part[i] = __fmul_rn(y[i], y[i]);
        const int lane = tid & 31;
#pragma unroll
        for (int off = 16, held = PT_TOKENS / 2; off > 1; off >>= 1, held >>= 1) {
            const bool high = lane & off;
#pragma unroll
            for (int k = 0; k < PT_TOKENS / 2; ++k)
                if (k < held) {
                    const float send = high ? part[k] : part[k + held], keep = high ? part[k + held] : part[k];
                    part[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
        }
        part[0] += __shfl_xor_sync(0xffffffffu, part[0], 1);
        if (!(lane & 1)) red[tid >> 5][lane >> 1] = part[0];
        __syncthreads();
        const bool is_q = unit < kv_heads;
        if (tid < PT_TOKENS) {  // (a token's factor once, over one of the sums that this thread alone reads)
            float f = 1.0f / sqrtf(((red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid])) + 1e-6f);
            if (is_q) f *= 1.0f / sqrtf((float)dim);
            red[0][tid] = f;
        }
        __syncthreads();
        float* dst = (is_q ? q_out : k_out) + (size_t)n0 * qk + (is_q ? unit : unit - kv_heads) * dim + i0;
#pragma unroll
        for (int i = 0; i < PT_TOKENS; ++i) {
            if (live && i < cnt) dst[(size_t)i * qk] = y[i] * red[0][i];
        }
    }
}

// The same where channels come in aligned pieces of four: a warp per unit and 8 tokens, a lane four neighbouring channels.  Rows of the block
// and those before it go to shared memory, all on their way at once, and every lane reads what it fetched itself: no barriers, no
// registers that wait for memory, little code.  The exponentials and divisions bound it (27 million instructions here, 41 there), then
// the warps in flight.  (2,048 tokens of 16 heads of 128 x 128: the kernel above 57 us, this one 45, with 16 tokens a warp and half as many
// warps an SM 56; 4,000 tokens of 32 heads on 16 150 and 111; the bytes of the first take 20.)  Every number is the same chain of operations as
// above, also the sums of squares: a token's results do not depend on how many others the step has.
constexpr int PW_TOKENS = 8, PW_LD = 128 + 4;  // (rows so far apart that eight tokens' pieces of one column meet in no bank)
template <int TAPS> constexpr int pw_floats() { return (PW_TOKENS + TAPS - 1) * PW_LD; }
template <int TAPS>
__global__ void __launch_bounds__(128)
delta_prep_warp_kernel(const float* __restrict__ qkvb, int ld, const float* __restrict__ a, const float* __restrict__ conv_w,
                       const float* __restrict__ A_log, const float* __restrict__ dt_bias, const float* __restrict__ state,
                       long long state_stride, const int* __restrict__ slots, const int* __restrict__ seq_of_token,
                       const int* __restrict__ cu_q, float* __restrict__ q_out, float* __restrict__ k_out, float* __restrict__ v_out,
                       float* __restrict__ beta, float* __restrict__ decay, int num_tokens, int heads, int kv_heads, int dim, int vdim,
                       int num_slots, int* err) {
    extern __shared__ __align__(16) float pw_smem[];
    ie_pdl_trigger();
    ie_pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, unit = blockIdx.y * 4 + warp;
    const int n0 = blockIdx.x * PW_TOKENS, cnt = min(PW_TOKENS, num_tokens - n0), qk = kv_heads * dim, channels = 2 * qk + heads * vdim;
    float* rows = pw_smem + warp * pw_floats<TAPS>();  // [PW_TOKENS + TAPS - 1][128 + 4]
    auto bring = [&](int row, const float* src) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(rows + row * PW_LD + lane * 4)), "l"(src) : "memory");
    };
    if (unit > 2 * kv_heads + 2 * heads) return;
    if (unit == 2 * kv_heads + 2 * heads) {  // the betas
        for (int i = lane; i < cnt * heads; i += 32) {
            const size_t n = (size_t)(n0 + i / heads);
            beta[n * heads + i % heads] = sigmoid_f(qkvb[n * ld + channels + i % heads]);
        }
        return;
    }
    const bool is_decay = unit >= 2 * kv_heads + heads, is_v = unit >= 2 * kv_heads && !is_decay;
    const int width = is_v ? vdim : dim;
    // the block's tokens, one a lane: its place in its request, and the slot
    int t_of = 0, slot_of = 0;
    if (!is_decay && lane < cnt) {
        const int seq = seq_of_token[n0 + lane];
        t_of = n0 + lane - cu_q[seq];
        slot_of = slots[seq];
        if (slot_of < 0 || slot_of >= num_slots) {
            ie_report(err, IE_ERR_PAGE, slot_of, n0 + lane);
            slot_of = -1;
        }
    }
    for (int c0 = 0; c0 < width; c0 += 128) {  // (q, k and decays: once)
        const int i0 = c0 + lane * 4;
        const bool live = i0 < width;
        if (is_decay) {
            const int h = unit - 2 * kv_heads - heads;
            const size_t at = (size_t)n0 * heads * dim + h * dim + i0, step = (size_t)heads * dim;
            if (live)
                for (int i = 0; i < cnt; ++i) bring(i, a + at + i * step);
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (!live) continue;
            const float rate = expf(A_log[h]);
            const float4 b = *reinterpret_cast<const float4*>(dt_bias + h * dim + i0);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll 2
            for (int i = 0; i < cnt; ++i) {
                const float4 x = *reinterpret_cast<const float4*>(rows + i * PW_LD + lane * 4);
                *reinterpret_cast<float4*>(decay + at + i * step) =
                    make_float4(expf(-rate * softplus_f(x.x + b.x)), expf(-rate * softplus_f(x.y + b.y)),
                                expf(-rate * softplus_f(x.z + b.z)), expf(-rate * softplus_f(x.w + b.w)));
            }
            continue;
        }
        const int c = (is_v ? 2 * qk + (unit - 2 * kv_heads) * vdim : unit * dim) + i0;
        if (live)
            for (int i = 0; i < cnt + TAPS - 1; ++i)
                if (n0 + i >= TAPS - 1) bring(i, qkvb + (size_t)(n0 + i - (TAPS - 1)) * ld + c);
        asm volatile("cp.async.commit_group;" ::: "memory");
        float w[4][TAPS];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int j = 0; j < TAPS; ++j) w[e][j] = live ? conv_w[(size_t)(c + e) * TAPS + j] : 0.f;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll 2
        for (int i = 0; i < cnt; ++i) {
            const int t = __shfl_sync(0xffffffffu, t_of, i), slot = __shfl_sync(0xffffffffu, slot_of, i);
            float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && slot >= 0) {
                float4 x[TAPS];
#pragma unroll
                for (int j = 0; j < TAPS; ++j) x[j] = *reinterpret_cast<const float4*>(rows + (i + j) * PW_LD + lane * 4);
                if (t < TAPS - 1) {  // the first look back to the kept ones
                    const float* tail = state + (size_t)slot * state_stride + (size_t)heads * dim * vdim + c;
#pragma unroll
                    for (int j = 0; j < TAPS - 1; ++j)
                        if (t + j < TAPS - 1) {
                            const float* kept = tail + (size_t)(t + j) * channels;
                            x[j] = make_float4(kept[0], kept[1], kept[2], kept[3]);
                        }
                }
#pragma unroll
                for (int j = 0; j < TAPS; ++j) {
                    y.x = fmaf(w[0][j], x[j].x, y.x);
                    y.y = fmaf(w[1][j], x[j].y, y.y);
                    y.z = fmaf(w[2][j], x[j].z, y.z);
                    y.w = fmaf(w[3][j], x[j].w, y.w);
                }
                y = make_float4(silu_f(y.x), silu_f(y.y), silu_f(y.z), silu_f(y.w));
            }
            if (is_v) {
                if (live) *reinterpret_cast<float4*>(v_out + (size_t)(n0 + i) * heads * vdim + (c - 2 * qk)) = y;
            } else {
                *reinterpret_cast<float4*>(rows + i * PW_LD + lane * 4) = y;  // (a row that no later token looks back to)
            }
        }
        if (is_v) continue;
        // The squares of a token's 32 channels per lane (channel d's with d + 16, then with d + 8 and so on, as a warp of the kernels above adds
        // them), the four sums of 32, then the token's factor.
        __syncwarp();
        float part[32];
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
            const float4 y = *reinterpret_cast<const float4*>(rows + lane % PW_TOKENS * PW_LD + lane / PW_TOKENS * 32 + k);
            part[k] = __fmul_rn(y.x, y.x);
            part[k + 1] = __fmul_rn(y.y, y.y);
            part[k + 2] = __fmul_rn(y.z, y.z);
            part[k + 3] = __fmul_rn(y.w, y.w);
        }
#pragma unroll
        for (int half = 16; half > 0; half >>= 1)
#pragma unroll
            for (int k = 0; k < half; ++k) part[k] += part[k + half];
        float sum = part[0];
        sum += __shfl_xor_sync(0xffffffffu, sum, PW_TOKENS);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2 * PW_TOKENS);
        float f = 1.0f / sqrtf(sum + 1e-6f);
        if (unit < kv_heads) f *= 1.0f / sqrtf((float)dim);
        float* dst = (unit < kv_heads ? q_out : k_out) + (size_t)n0 * qk + (unit < kv_heads ? unit : unit - kv_heads) * dim + i0;
#pragma unroll 4
        for (int i = 0; i < cnt; ++i) {
            const float factor = __shfl_sync(0xffffffffu, f, i);
            if (!live) continue;
            const float4 y = *reinterpret_cast<const float4*>(rows + i * PW_LD + lane * 4);
            *reinterpret_cast<float4*>(dst + (size_t)i * qk) = make_float4(y.x * factor, y.y * factor, y.z * factor, y.w * factor);
        }
    }
}

// grid: (requests of the step, blocks of 256 channels): the kept inputs become the last taps - 1 of (kept, new).  A thread owns a
// channel; with up to four kept rows every value is read before the first is written, so the reads wait for memory together.
__global__ void delta_conv_tail_kernel(const float* __restrict__ qkvb, int ld, float* __restrict__ state,
                                       long long state_stride, const int* __restrict__ slots,
                                       const int* __restrict__ cu_q, long long matrix_floats, int channels,
                                       int taps, int num_slots) {
    ie_pdl_trigger();
    ie_pdl_wait();
    int seq = blockIdx.x;
    int start = cu_q[seq], len = cu_q[seq + 1] - start;
    int slot = slots[seq], c = blockIdx.y * blockDim.x + threadIdx.x;
    if (len <= 0 || slot < 0 || slot >= num_slots || c >= channels) return;
    float* tail = state + (size_t)slot * state_stride + matrix_floats;
    // row j takes the input at step-relative time len - (taps - 1) + j
    auto kept = [&](int j) {
        int tt = len - (taps - 1) + j;
        return tt >= 0 ? qkvb[(size_t)(start + tt) * ld + c] : tail[(size_t)(taps - 1 + tt) * channels + c];
    };
    constexpr int MOST = 4;
    if (taps - 1 <= MOST) {
        float v[MOST];
#pragma unroll
        for (int j = 0; j < MOST; ++j)
            if (j < taps - 1) v[j] = kept(j);
#pragma unroll
        for (int j = 0; j < MOST; ++j)
            if (j < taps - 1) tail[(size_t)j * channels + c] = v[j];
        return;
    }
    for (int j = 0; j < taps - 1; ++j) tail[(size_t)j * channels + c] = kept(j);  // (rising: read before it is overwritten)
}

constexpr int DR_THREADS = 128;
constexpr int DR_CHUNK = 8;  // tokens staged in shared memory at a time

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async16f(float* dst, const float* src) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// grid: (column blocks, heads, requests).  R rows per lane; TPC lanes per column (a power of two).
// The tokens' k, q, decay, v and beta come through shared memory eight tokens at a time, the next
// eight on their way (cp.async, two buffers) while these are worked on.  A lane holds R (8 or 16)
// consecutive rows of its column; in shared memory a token's k, q and decay lie in groups of R
// entries R + 4 floats apart, so that a lane fetches its rows with 16-byte loads and the lanes of a
// column hit different banks; entries beyond `dim` read as zero, so the inner loops carry no bounds checks.
template <int R, int TPC>
__global__ void __launch_bounds__(DR_THREADS)
delta_rule_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                  const float* __restrict__ beta, const float* __restrict__ decay, float* __restrict__ state,
                  long long state_stride, const int* __restrict__ slots, const int* __restrict__ cu_q,
                  float* __restrict__ out, int heads, int kv_heads, int dim, int vdim, int num_slots) {
    extern __shared__ __align__(16) float sm[];  // two buffers of: k, q, g [CHUNK][DP] each, v [CHUNK][COLS], beta [CHUNK]
    static_assert(R == 8 || R == 16, "a lane's rows are one group of 8 or 16");
    constexpr int GS = R + 4;  // a lane's group of R entries, and four floats to the next lane's
    constexpr int COLS = DR_THREADS / TPC, DP = GS * TPC;  // a token's row of k (q, decay)
    constexpr int BUF = DR_CHUNK * (3 * DP + COLS + 4);
    ie_pdl_trigger();
    ie_pdl_wait();
    int seq = blockIdx.z, head = blockIdx.y;
    int start = cu_q[seq], len = cu_q[seq + 1] - start;
    int slot = slots[seq];
    if (len <= 0 || slot < 0 || slot >= num_slots) return;
    int tid = threadIdx.x;
    int sub = tid % TPC, my_col = tid / TPC, col = blockIdx.x * COLS + my_col;
    bool live = col < vdim;
    int kvh = head / (heads / kv_heads);
    float* S = state + (size_t)slot * state_stride + ((size_t)head * vdim + (live ? col : 0)) * dim;
    float s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        int r = sub * R + i;
        s[i] = (live && r < dim) ? S[r] : 0.f;
    }
    // what the copies never touch (entries beyond dim, the gaps) reads as zero
    for (int i = tid; i < 2 * BUF; i += DR_THREADS) sm[i] = 0.f;
    __syncthreads();
    int c0 = blockIdx.x * COLS;
    bool vec = (dim % 4 == 0) && (vdim % 4 == 0) && (COLS % 4 == 0);
    auto stage = [&](int t0, int b) {  // the chunk's values on their way into buffer b
        int cnt = min(DR_CHUNK, len - t0);
        float* ks = sm + b * BUF;
        float* qs = ks + DR_CHUNK * DP;
        float* gs = qs + DR_CHUNK * DP;
        float* vs = gs + DR_CHUNK * DP;
        float* bs = vs + DR_CHUNK * COLS;
        if (vec) {  // rows and column runs of whole 16-byte pieces
            int dq = dim >> 2;
            for (int i = tid; i < cnt * dq; i += DR_THREADS) {
                int tt = i / dq, d = (i - tt * dq) * 4;
                size_t n = (size_t)(start + t0 + tt);
                int at = tt * DP + (d / R) * GS + (d % R);
                cp_async16f(ks + at, k + (n * kv_heads + kvh) * dim + d);
                cp_async16f(qs + at, q + (n * kv_heads + kvh) * dim + d);
                cp_async16f(gs + at, decay + (n * heads + head) * dim + d);
            }
            for (int i = tid; i < cnt * (COLS / 4); i += DR_THREADS) {
                int tt = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
                if (c0 + c < vdim) cp_async16f(vs + tt * COLS + c, v + ((size_t)(start + t0 + tt) * heads + head) * vdim + c0 + c);
            }
        } else {
            for (int tt = 0; tt < cnt; ++tt) {
                size_t n = (size_t)(start + t0 + tt);
                for (int d = tid; d < dim; d += DR_THREADS) {
                    int at = tt * DP + (d / R) * GS + (d % R);
                    cp_async4(ks + at, k + (n * kv_heads + kvh) * dim + d);
                    cp_async4(qs + at, q + (n * kv_heads + kvh) * dim + d);
                    cp_async4(gs + at, decay + (n * heads + head) * dim + d);
                }
                if (tid < COLS && c0 + tid < vdim) cp_async4(vs + tt * COLS + tid, v + (n * heads + head) * vdim + c0 + tid);
            }
        }
        if (tid < cnt) cp_async4(bs + tid, beta + (size_t)(start + t0 + tid) * heads + head);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, 0);
    int b = 0;
    for (int t0 = 0; t0 < len; t0 += DR_CHUNK, b ^= 1) {
        int cnt = min(DR_CHUNK, len - t0);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this chunk has landed for everyone, and everyone is done with the other buffer
        if (t0 + DR_CHUNK < len) stage(t0 + DR_CHUNK, b ^ 1);
        const float* ks = sm + b * BUF + sub * GS;
        const float* qs = ks + DR_CHUNK * DP;
        const float* gs = qs + DR_CHUNK * DP;
        const float* vs = sm + b * BUF + 3 * DR_CHUNK * DP + my_col;
        const float* bs = sm + b * BUF + 3 * DR_CHUNK * DP + DR_CHUNK * COLS;
        for (int tt = 0; tt < cnt; ++tt) {
            const float* kt = ks + tt * DP;
            const float* qt = qs + tt * DP;
            const float* gt = gs + tt * DP;
            float kv[R], gv[R], qv[R];
#pragma unroll
            for (int j = 0; j < R / 4; ++j) {
                *reinterpret_cast<float4*>(kv + 4 * j) = reinterpret_cast<const float4*>(kt)[j];
                *reinterpret_cast<float4*>(gv + 4 * j) = reinterpret_cast<const float4*>(gt)[j];
                *reinterpret_cast<float4*>(qv + 4 * j) = reinterpret_cast<const float4*>(qt)[j];
            }
            float d4[4] = {0.f, 0.f, 0.f, 0.f};  // four partial sums: shorter chains, a fixed order
#pragma unroll
            for (int i = 0; i < R; ++i) {
                s[i] *= gv[i];
                d4[i & 3] = fmaf(s[i], kv[i], d4[i & 3]);
            }
            float dot = (d4[0] + d4[1]) + (d4[2] + d4[3]);
#pragma unroll
            for (int o = TPC >> 1; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            float u = bs[tt] * ((live ? vs[tt * COLS] : 0.f) - dot);
            float r4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < R; ++i) {
                s[i] = fmaf(kv[i], u, s[i]);
                r4[i & 3] = fmaf(s[i], qv[i], r4[i & 3]);
            }
            float rd = (r4[0] + r4[1]) + (r4[2] + r4[3]);
#pragma unroll
            for (int o = TPC >> 1; o > 0; o >>= 1) rd += __shfl_xor_sync(0xffffffffu, rd, o);
            if (live && sub == 0) out[((size_t)(start + t0 + tt) * heads + head) * vdim + col] = rd;
        }
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            int r = sub * R + i;
            if (r < dim) S[r] = s[i];
        }
    }
}

// One warp per (token, head).
template <typename T>
__global__ void __launch_bounds__(128)
gated_rms_heads_kernel(const float* __restrict__ o, const float* __restrict__ weight, float eps,
                       const float* __restrict__ gate_pre, T* __restrict__ out, long long rows, int vdim) {
    ie_pdl_trigger();
    ie_pdl_wait();
    long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= rows) return;
    int lane = threadIdx.x & 31;
    const float* src = o + row * vdim;
    float ss = 0.f;
    for (int d = lane; d < vdim; d += 32) ss = fmaf(src[d], src[d], ss);
    ss = warp_sum(ss);
    float inv = 1.0f / sqrtf(ss / (float)vdim + eps);
    for (int d = lane; d < vdim; d += 32)
        ie_store(out + row * vdim + d, src[d] * inv * weight[d] * sigmoid_f(gate_pre[row * vdim + d]));
}
}  // namespace

IE_API int ie_delta_prep(const float* qkvb, int ld, const float* a, const float* conv_w, const float* A_log,
                         const float* dt_bias, float* state, long long state_stride, const int* slots,
                         const int* seq_of_token, const int* cu_q, float* q_out, float* k_out, float* v_out,
                         float* beta, float* decay, int num_tokens, int num_seqs, int heads, int kv_heads,
                         int dim, int vdim, int taps, int num_slots, int* err, void* stream) {
    if (num_tokens <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    size_t smem = (size_t)(dim > vdim ? dim : vdim) * sizeof(float);
    if (smem > 48 * 1024) return (int)cudaErrorInvalidValue;
    int units = 2 * kv_heads + 2 * heads + 1, e;
    const dim3 tiles((num_tokens + PT_TOKENS - 1) / PT_TOKENS, units);
#define IE_DP_TILE(TAPS)                                                                                               \
    e = ie_launch(delta_prep_tile_kernel<TAPS>, tiles, dim3(128), 0, s, qkvb, ld, a, conv_w, A_log, dt_bias,           \
                  (const float*)state, state_stride, slots, seq_of_token, cu_q, q_out, k_out, v_out, beta, decay,      \
                  num_tokens, heads, kv_heads, dim, vdim, num_slots, err)
#define IE_DP_WARP(TAPS)                                                                                               \
    {                                                                                                                  \
        static IePerDevice allowed;                                                                                    \
        cudaError_t e2 = ie_allow_smem(allowed, delta_prep_warp_kernel<TAPS>, 4 * pw_floats<TAPS>() * sizeof(float));  \
        if (e2 != cudaSuccess) return (int)e2;                                                                         \
        e = ie_launch(delta_prep_warp_kernel<TAPS>, dim3((num_tokens + PW_TOKENS - 1) / PW_TOKENS, (units + 3) / 4), dim3(128), 4 * pw_floats<TAPS>() * sizeof(float), \
                      s, qkvb, ld, a, conv_w, A_log, dt_bias, (const float*)state, state_stride, slots, seq_of_token, cu_q, q_out, \
                      k_out, v_out, beta, decay, num_tokens, heads, kv_heads, dim, vdim, num_slots, err);              \
    }
    // (from 64 tokens on the tiles are enough blocks to fill the device; a few tokens get a block per token and unit)
    const bool tile = num_tokens >= 64 && dim <= 128;
    // (a warp per unit and 8 tokens from 256 tokens on: 128 tokens of 16 heads of 128 x 128 8.6 us in tiles, 9.6 so, 256 of 8 heads of 64 x 64
    // 9.7 and 8.8)
    const bool fours = tile && num_tokens >= 256 && dim % 4 == 0 && vdim % 4 == 0 && ld % 4 == 0 &&
                       !(((size_t)qkvb | (size_t)a | (size_t)dt_bias | (size_t)q_out | (size_t)k_out | (size_t)v_out | (size_t)decay) & 15);
    if (fours && taps == 4) IE_DP_WARP(4)
    else if (fours && taps == 3) IE_DP_WARP(3)
    else if (fours && taps == 2) IE_DP_WARP(2)
    else if (tile && taps == 4) IE_DP_TILE(4);
    else if (tile && taps == 3) IE_DP_TILE(3);
    else if (tile && taps == 2) IE_DP_TILE(2);
    else
        e = ie_launch(delta_prep_kernel, dim3(num_tokens, num_tokens >= 512 ? (units < 4 ? units : 4) : units), dim3(128), smem, s,
                      qkvb, ld, a, conv_w, A_log, dt_bias, (const float*)state, state_stride, slots, seq_of_token, cu_q, q_out,
                      k_out, v_out, beta, decay, heads, kv_heads, dim, vdim, taps, num_slots, err);
#undef IE_DP_TILE
#undef IE_DP_WARP
    if (e != 0 || taps < 2) return e;
    int channels = 2 * kv_heads * dim + heads * vdim;
    return ie_launch(delta_conv_tail_kernel, dim3(num_seqs, (channels + 255) / 256), dim3(256), 0, s, qkvb, ld, state, state_stride, slots,
                     cu_q, (long long)heads * dim * vdim, channels, taps, num_slots);
}

template <int R, int TPC>
static int launch_delta_rule(const float* q, const float* k, const float* v, const float* beta, const float* decay,
                             float* state, long long state_stride, const int* slots, const int* cu_q, float* out,
                             int num_seqs, int heads, int kv_heads, int dim, int vdim, int num_slots, cudaStream_t s) {
    constexpr int COLS = DR_THREADS / TPC;
    size_t smem = (size_t)2 * DR_CHUNK * (3 * (R + 4) * TPC + COLS + 4) * sizeof(float);
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, delta_rule_kernel<R, TPC>, 160 * 1024);  // (dim 512: 124 KB)
    if (e != cudaSuccess) return (int)e;
    dim3 grid((vdim + COLS - 1) / COLS, heads, num_seqs);
    return ie_launch(delta_rule_kernel<R, TPC>, grid, dim3(DR_THREADS), smem, s, q, k, v, beta, decay, state,
                     state_stride, slots, cu_q, out, heads, kv_heads, dim, vdim, num_slots);
}

IE_API int ie_delta_rule(const float* q, const float* k, const float* v, const float* beta, const float* decay,
                         float* state, long long state_stride, const int* slots, const int* cu_q, float* out,
                         int num_seqs, int heads, int kv_heads, int dim, int vdim, int num_slots, void* stream) {
    if (num_seqs <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
#define IE_DR_ARGS q, k, v, beta, decay, state, state_stride, slots, cu_q, out, num_seqs, heads, kv_heads, dim, vdim, num_slots, s
    // Eight rows per lane for small key sizes (2,048 tokens of 8 heads of 64 x 64: 0.54 ms against 0.65 with
    // sixteen), sixteen from there on (16 heads of 128 x 128: 0.64 ms against 0.75 with eight: the exchange
    // between a column's lanes has a step more).
    if (dim <= 8) return launch_delta_rule<8, 1>(IE_DR_ARGS);
    if (dim <= 16) return launch_delta_rule<8, 2>(IE_DR_ARGS);
    if (dim <= 32) return launch_delta_rule<8, 4>(IE_DR_ARGS);
    if (dim <= 64) return launch_delta_rule<8, 8>(IE_DR_ARGS);
    if (dim <= 128) return launch_delta_rule<16, 8>(IE_DR_ARGS);
    if (dim <= 256) return launch_delta_rule<16, 16>(IE_DR_ARGS);
    if (dim <= 512) return launch_delta_rule<16, 32>(IE_DR_ARGS);
#undef IE_DR_ARGS
    return (int)cudaErrorInvalidValue;  // dim <= 512
}

IE_API int ie_gated_rms_heads(const float* o, const float* weight, float eps, const float* gate_pre, void* out,
                              int out_dtype, long long rows, int vdim, void* stream) {
    if (rows <= 0) return 0;
    dim3 grid((unsigned)((rows + 3) / 4));
    cudaStream_t s = (cudaStream_t)stream;
    if (gated_rows_fit(o, weight, gate_pre, vdim, out, rows, vdim))
        return out_dtype == IE_BF16 ? launch_gated_rows(o, weight, 0, eps, gate_pre, vdim, 0, (__nv_bfloat16*)out, rows, 1, vdim, s)
                                    : launch_gated_rows(o, weight, 0, eps, gate_pre, vdim, 0, (float*)out, rows, 1, vdim, s);
    if (out_dtype == IE_BF16)
        return ie_launch(gated_rms_heads_kernel<__nv_bfloat16>, grid, dim3(128), 0, s, o, weight, eps, gate_pre,
                         (__nv_bfloat16*)out, rows, vdim);
    return ie_launch(gated_rms_heads_kernel<float>, grid, dim3(128), 0, s, o, weight, eps, gate_pre, (float*)out,
                     rows, vdim);
}
