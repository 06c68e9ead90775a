// Rows that are divided by their root mean square, weighted and gated, in aligned pieces of four.
#pragma once
#include "common.cuh"

namespace {

constexpr int GR_ROWS = 2, GR_MOST = 128;

__device__ __forceinline__ void gr_store(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void gr_store(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
}

// The sum of a row's squares, entries 4 lane .. + 3 in x, as it comes from lanes that hold every 32nd entry: each its own in order, then warp_sum.
// Lane 8 j + a gets entry 4 a + j of every 32; of their number in 32 lane bits 2, 1, 0 then are bits 4, 3, 2 and lane bits 4, 3 bits 1, 0.
__device__ __forceinline__ float gr_sum_of_squares(float4 x, int lane) {
    float v[4] = {x.x, x.y, x.z, x.w};  // a 4 x 4 square over lanes a, 8 + a, 16 + a, 24 + a, turned over: by twos, then by ones
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const bool high = lane & 16;
        const float other = __shfl_xor_sync(0xffffffffu, high ? v[k] : v[k + 2], 16);
        if (high) v[k] = other;
        else v[k + 2] = other;
    }
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        const bool high = lane & 8;
        const float other = __shfl_xor_sync(0xffffffffu, high ? v[k] : v[k + 1], 8);
        if (high) v[k] = other;
        else v[k + 1] = other;
    }
    float s = fmaf(v[3], v[3], fmaf(v[2], v[2], fmaf(v[1], v[1], fmaf(v[0], v[0], 0.f))));
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    return s;
}

// A row per (token, head) of up to 128 values; a lane four neighbouring ones, a warp GR_ROWS rows, whose loads are on their way together.
// Every number is the same chain of operations as in the kernels that hold every 32nd entry in a lane, so a row's result does not depend on how many there are:
// before the sum of squares the lanes exchange entries so that each has those.
// weight: [vdim], or [heads * vdim], or null; gate_pre: element (n, head, d) at [n * gate_ld + head * vdim + d], or null.  Memory
// bounds it.  (2,048 tokens of 16 heads of 128 with gates, into bfloat16, 42 MB: 15.4 us with an entry a lane at a time and a row a warp, 11.4 so.)
template <typename T>
__global__ void __launch_bounds__(128)
gated_rows_kernel(const float* __restrict__ o, const float* __restrict__ weight, int weight_per_head, float eps,
                  const float* __restrict__ gate_pre, int gate_ld, int gate_silu, T* __restrict__ out, long long rows, int heads, int vdim) {
    ie_pdl_trigger();
    ie_pdl_wait();
    const long long first = ((long long)blockIdx.x * 4 + (threadIdx.x >> 5)) * GR_ROWS;
    const int lane = threadIdx.x & 31, d = lane * 4;
    float4 x[GR_ROWS], g[GR_ROWS], w[GR_ROWS];
#pragma unroll
    for (int r = 0; r < GR_ROWS; ++r) {
        const long long row = first + r, n = row / heads;
        const int head = (int)(row - n * heads);
        const bool in = row < rows && d < vdim;
        x[r] = g[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        w[r] = make_float4(1.f, 1.f, 1.f, 1.f);
        if (in) x[r] = *reinterpret_cast<const float4*>(o + row * vdim + d);
        if (in && gate_pre != nullptr) g[r] = *reinterpret_cast<const float4*>(gate_pre + n * gate_ld + (size_t)head * vdim + d);
        if (in && weight != nullptr) w[r] = *reinterpret_cast<const float4*>(weight + (weight_per_head ? (size_t)head * vdim : 0) + d);
    }
#pragma unroll
    for (int r = 0; r < GR_ROWS; ++r) {
        const float inv = 1.0f / sqrtf(gr_sum_of_squares(x[r], lane) / (float)vdim + eps);
        const float xs[4] = {x[r].x, x[r].y, x[r].z, x[r].w}, gs[4] = {g[r].x, g[r].y, g[r].z, g[r].w}, ws[4] = {w[r].x, w[r].y, w[r].z, w[r].w};
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            y[e] = xs[e] * inv;
            if (weight != nullptr) y[e] *= ws[e];
            if (gate_pre != nullptr) y[e] *= (gate_silu ? gs[e] : 1.0f) / (1.0f + expf(-gs[e]));
        }
        if (first + r < rows && d < vdim) gr_store(out + (first + r) * vdim + d, make_float4(y[0], y[1], y[2], y[3]));
    }
}

// Whether a call's rows and addresses allow it, and enough rows that a warp may take several.
inline bool gated_rows_fit(const void* o, const void* weight, const void* gate_pre, int gate_ld, const void* out, long long rows, int vdim) {
    return vdim % 4 == 0 && vdim <= GR_MOST && gate_ld % 4 == 0 && !(((size_t)o | (size_t)weight | (size_t)gate_pre | (size_t)out) & 15) &&
           rows >= 16ll * ie_sm_count();
}
template <typename T>
int launch_gated_rows(const float* o, const float* weight, int weight_per_head, float eps, const float* gate_pre, int gate_ld, int gate_silu,
                      T* out, long long rows, int heads, int vdim, cudaStream_t s) {
    const dim3 grid((unsigned)((rows + 4 * GR_ROWS - 1) / (4 * GR_ROWS)));
    return ie_launch(gated_rows_kernel<T>, grid, dim3(128), 0, s, o, weight, weight_per_head, eps, gate_pre, gate_ld, gate_silu, out, rows, heads, vdim);
}

}  // namespace
