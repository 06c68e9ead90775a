// Kernels of the latent attention mixer besides the attention itself (which is the general paged
// kernel with value rows inside the key rows, or the tensor-core kernel of latent_attention_mma.cu):
//
//  * latent_prep: from the 32-bit products of the mixer's input, per token, whichever of these are asked for:
//    the queries' unrotated parts and their rotated parts (turned, written behind the latent part of the
//    query rows the attention reads); the heads' output gates; the cached row: the latent (divided by
//    its root mean square, times a weight) followed by the shared rotated key part; the queries' own
//    latent (divided by its root mean square, times a weight), from which another product makes the queries.
//  * headwise_linear: out[n, h, :] = W[h] x[n, h, :] (times an optional factor per token and
//    head): the products that move the per-head key and value matrices to the query side.
//  * headwise_mma: the same on the tensor cores (bfloat16) for steps of up to some hundred tokens; it can
//    read the 32-bit queries themselves and turn their rotated parts on the way, so that a step that follows
//    the queries' product needs one launch for everything up to the attention.
//
// Rotation of the first rot_dims entries of the rotated part, a = position * frequency from the 32-bit table
// [positions, 2, rot_dims / 2] (cosines, then sines, with whatever factor the encoding has): entries 2i and
// 2i+1 form a pair, or (halves) entries i and i + rot_dims / 2; (u, v) -> (u cos a - v sin a, v cos a + u sin a);
// entries from rot_dims on pass unchanged.
// All arithmetic is 32-bit; results are rounded once to the output's dtype.
#include "common.cuh"

namespace {

// A row of a 32-bit product that may have come back in parts (of a split inner dimension): added in order.
struct Row {
    const float* p;
    int parts;
    size_t stride;
    __device__ __forceinline__ float operator[](int i) const {
        float v = p[i];
#pragma unroll 4
        for (int s = 1; s < parts; ++s) v += p[s * stride + i];
        return v;
    }
    __device__ __forceinline__ float4 four(int i) const {
        float4 v = *reinterpret_cast<const float4*>(p + i);
#pragma unroll 8
        for (int s = 1; s < parts; ++s) {
            float4 x = *reinterpret_cast<const float4*>(p + s * stride + i);
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        return v;
    }
    __device__ __forceinline__ Row at(int i) const { return Row{p + i, parts, stride}; }
};

// entry d of a rotated part `src`, turned by the angles at `cs` (null: not turned)
template <typename Src>
__device__ __forceinline__ float turned(const Src& src, int d, const float* cs, int rot_dims, int interleaved) {
    float v = src[d];
    if (cs == nullptr || d >= rot_dims) return v;
    int half = rot_dims / 2;
    int j = interleaved ? d >> 1 : (d < half ? d : d - half);
    bool second = interleaved ? (d & 1) != 0 : d >= half;
    float c = cs[j], s = cs[half + j];
    if (second) return fmaf(v, c, src[interleaved ? d - 1 : d - half] * s);
    return fmaf(v, c, -src[interleaved ? d + 1 : d + half] * s);
}

// Entries d .. d + 3 of the same, of a row in one part (rot_dims, and half of it where entries half apart form pairs, multiples of 4).
__device__ __forceinline__ float4 turned4(const float* src, int d, const float* cs, int rot_dims, int interleaved) {
    const float4 v = *reinterpret_cast<const float4*>(src + d);
    if (cs == nullptr || d >= rot_dims) return v;
    const int half = rot_dims / 2;
    if (interleaved) {
        const float2 c = *reinterpret_cast<const float2*>(cs + d / 2), s = *reinterpret_cast<const float2*>(cs + half + d / 2);
        return make_float4(fmaf(v.x, c.x, -v.y * s.x), fmaf(v.y, c.x, v.x * s.x), fmaf(v.z, c.y, -v.w * s.y), fmaf(v.w, c.y, v.z * s.y));
    }
    const int j = d >= half ? d - half : d;
    const float sign = d >= half ? 1.f : -1.f;
    const float4 o = *reinterpret_cast<const float4*>(src + (d >= half ? j : d + half)), c = *reinterpret_cast<const float4*>(cs + j);
    const float4 s = *reinterpret_cast<const float4*>(cs + half + j);
    return make_float4(fmaf(v.x, c.x, sign * o.x * s.x), fmaf(v.y, c.y, sign * o.y * s.y), fmaf(v.z, c.z, sign * o.z * s.z), fmaf(v.w, c.w, sign * o.w * s.w));
}

__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    __nv_bfloat162 o[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
    *reinterpret_cast<uint2*>(p) = *reinterpret_cast<uint2*>(o);
}

// What a call asks for is what has a pointer: queries (q), gates (gate_pre), the cached row (dkv and
// slot_mapping), the queries' latent (cq).  Each input is a row `*_ld` numbers long per token, in `parts` parts
// `part_stride` apart.
struct LatentIn {
    const float* q; int q_ld;
    const float* gate_pre; int gate_ld;
    const float* dkv; int dkv_ld;
    const float* cq; int cq_ld, q_rank;
    int parts; size_t part_stride;
    const float* norm_w;
    const float* cq_norm_w;
    float eps;
    bool fours;    // sizes and addresses of cq and dkv allow pieces of four
    bool all_fours;  // those of everything that is asked for, and the rotation
    __device__ Row row(const float* p, int ld, int n) const { return Row{p + (size_t)n * ld, parts, part_stride}; }
};

constexpr int LP_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(LP_THREADS)
latent_prep_kernel(LatentIn in, const int* __restrict__ positions,
                   const float* __restrict__ table, int rot_dims, int table_rows, int interleaved,
                   T* __restrict__ q_plain, T* __restrict__ q_abs, float* __restrict__ gate, T* __restrict__ cq_out,
                   T* __restrict__ cache, const int* __restrict__ slot_mapping, int heads, int dim, int rot_dim,
                   int rank, int total_slots, int* err) {
    extern __shared__ __align__(16) float rows[];  // the queries' latent, then the cached row, as they come
    __shared__ float red[2][LP_THREADS / 32];
    ie_pdl_trigger();
    ie_pdl_wait();
    int n = blockIdx.x, tid = threadIdx.x;
    int hq = dim + rot_dim, krow = rank + rot_dim;
    int pos = positions[n];
    bool turn = table != nullptr && rot_dims > 0;
    if (turn && (pos < 0 || pos >= table_rows)) {
        if (tid == 0) ie_report(err, IE_ERR_POSITION, pos, n);
        turn = false;
    }
    const float* cs = turn ? table + (size_t)pos * rot_dims : nullptr;  // cos [rot_dims/2], then sin

    if (in.q != nullptr) {
        // queries: unrotated parts as they are, rotated parts behind the latent part of the query rows
        const Row row = in.row(in.q, in.q_ld, n);
        for (int i = tid; i < heads * dim; i += LP_THREADS) {
            int h = i / dim, d = i - h * dim;
            ie_store(q_plain + (size_t)n * heads * dim + i, row[h * hq + d]);
        }
        for (int i = tid; i < heads * rot_dim; i += LP_THREADS) {
            int h = i / rot_dim, d = i - h * rot_dim;
            ie_store(q_abs + ((size_t)n * heads + h) * krow + rank + d, turned(row.at(h * hq + dim), d, cs, rot_dims, interleaved));
        }
    }
    if (in.gate_pre != nullptr) {
        const Row g = in.row(in.gate_pre, in.gate_ld, n);
        for (int h = tid; h < heads; h += LP_THREADS) gate[(size_t)n * heads + h] = 1.0f / (1.0f + expf(-g[h]));
    }
    int slot = in.dkv != nullptr && slot_mapping != nullptr ? slot_mapping[n] : -1;
    bool cached = in.dkv != nullptr && slot_mapping != nullptr;  // (a run that borrows another layer's cache writes none)
    if (cached && (slot < 0 || slot >= total_slots)) {
        if (tid == 0) ie_report(err, IE_ERR_PAGE, slot, n);
        cached = false;
    }
    const int n_cq = in.cq != nullptr ? in.q_rank : 0, n_row = cached ? krow : 0;
    if (n_cq + n_row == 0) return;
    const Row cq = in.row(in.cq, in.cq_ld, n), dkv = in.row(in.dkv, in.dkv_ld, n);
    float ss_q = 0.f, ss_c = 0.f;
    if (in.fours) {
#pragma unroll 2
        for (int i = tid * 4; i < n_cq + n_row; i += LP_THREADS * 4) {
            float4 v = i < n_cq ? cq.four(i) : dkv.four(i - n_cq);
            *reinterpret_cast<float4*>(rows + i) = v;
            float s = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w)));
            if (i < n_cq) ss_q += s;
            else if (i - n_cq < rank) ss_c += s;
        }
    } else {
        for (int i = tid; i < n_cq + n_row; i += LP_THREADS) {
            float v = i < n_cq ? cq[i] : dkv[i - n_cq];
            rows[i] = v;
            if (i < n_cq) ss_q = fmaf(v, v, ss_q);
            else if (i - n_cq < rank) ss_c = fmaf(v, v, ss_c);
        }
    }
    ss_q = warp_sum(ss_q);
    ss_c = warp_sum(ss_c);
    if ((tid & 31) == 0) { red[0][tid >> 5] = ss_q; red[1][tid >> 5] = ss_c; }
    __syncthreads();
    ss_q = ss_c = 0.f;
#pragma unroll
    for (int w = 0; w < LP_THREADS / 32; ++w) { ss_q += red[0][w]; ss_c += red[1][w]; }
    const float inv_q = n_cq > 0 ? 1.0f / sqrtf(ss_q / (float)n_cq + in.eps) : 0.f;
    const float inv_c = 1.0f / sqrtf(ss_c / (float)rank + in.eps);
    T* dst = cache + (size_t)max(slot, 0) * krow;
    const float* part = rows + n_cq + rank;
    for (int i = tid; i < n_cq + n_row; i += LP_THREADS) {
        if (i < n_cq) ie_store(cq_out + (size_t)n * n_cq + i, rows[i] * inv_q * in.cq_norm_w[i]);
        else if (i - n_cq < rank) ie_store(dst + i - n_cq, rows[i] * inv_c * in.norm_w[i - n_cq]);
        else ie_store(dst + i - n_cq, turned(part, i - n_cq - rank, cs, rot_dims, interleaved));
    }
}

// The sum of 256 threads' numbers as the kernel above adds them up, thread 32 w + lane's in s[w] of a lane: over every 32, by halves of them,
// then one 32 after the other.
__device__ __forceinline__ float block_order_sum(float (&s)[LP_THREADS / 32], int lane) {
    constexpr int WARPS = LP_THREADS / 32;
    static_assert(WARPS == 8, "");
#pragma unroll
    for (int off = 16, held = WARPS / 2; off > 0; off >>= 1, held >>= 1) {
        if (held > 0) {  // (every exchange halves the sums a lane still holds)
            const bool high = lane & off;
#pragma unroll
            for (int k = 0; k < WARPS / 2; ++k)
                if (k < held) {
                    const float send = high ? s[k] : s[k + held], keep = high ? s[k + held] : s[k];
                    s[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
        } else {
            s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
        }
    }
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) sum += __shfl_sync(0xffffffffu, s[0], 4 * w);
    return sum;
}

// The same for many tokens, of products in one part whose sizes and addresses allow pieces of four: a warp per token, no barriers, four of
// a lane's pieces on their way at a time.  Every number is the same chain of operations as there, also the sums of squares: a token's results do not depend on
// how many others the step has.  (2,048 tokens of 16 heads of 128 + 64 and a latent of 512: 28 us with a block per token and a launch each
// for the cached rows and the queries; 22 so with all of it beyond the L2, of which 2 are the order of the sums.  Most of the 28 was code fetched to be executed once, the sums over parts unrolled in
// every place: little code counts as much as few trips to memory here.)
constexpr int LW_WARPS = 4, LW_PIECES = 4;

template <typename T>
__global__ void __launch_bounds__(LW_WARPS * 32)
latent_prep_warp_kernel(LatentIn in, const int* __restrict__ positions, const float* __restrict__ table, int rot_dims, int table_rows,
                        int interleaved, T* __restrict__ q_plain, T* __restrict__ q_abs, float* __restrict__ gate, T* __restrict__ cq_out,
                        T* __restrict__ cache, const int* __restrict__ slot_mapping, int num_tokens, int heads, int dim, int rot_dim,
                        int rank, int total_slots, int* err) {
    ie_pdl_trigger();
    ie_pdl_wait();
    const int n = blockIdx.x * LW_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= num_tokens) return;
    const int hq = dim + rot_dim, krow = rank + rot_dim, pos = positions[n];
    const int slot = in.dkv != nullptr && slot_mapping != nullptr ? slot_mapping[n] : -1;
    bool turn = table != nullptr && rot_dims > 0, cached = in.dkv != nullptr && slot_mapping != nullptr;
    if (turn && (pos < 0 || pos >= table_rows)) {
        if (lane == 0) ie_report(err, IE_ERR_POSITION, pos, n);
        turn = false;
    }
    if (cached && (slot < 0 || slot >= total_slots)) {
        if (lane == 0) ie_report(err, IE_ERR_PAGE, slot, n);
        cached = false;
    }
    const float* cs = turn ? table + (size_t)pos * rot_dims : nullptr;
    if (in.gate_pre != nullptr)
        for (int h = lane; h < heads; h += 32) gate[(size_t)n * heads + h] = 1.0f / (1.0f + expf(-in.gate_pre[(size_t)n * in.gate_ld + h]));
    if (in.q != nullptr) {
        const float* row = in.q + (size_t)n * in.q_ld;
        for (int i0 = lane * 4; i0 < heads * hq; i0 += 128 * LW_PIECES) {
            float4 v[LW_PIECES];  // (all loads before the first store)
            T* to[LW_PIECES];
#pragma unroll
            for (int k = 0; k < LW_PIECES; ++k) {
                const int i = i0 + 128 * k, h = i / hq, d = i - h * hq;
                const bool plain = d < dim;
                to[k] = plain ? q_plain + ((size_t)n * heads + h) * dim + d : q_abs + ((size_t)n * heads + h) * krow + rank + d - dim;
                if (i < heads * hq) v[k] = turned4(row + i - d + dim, d - dim, plain ? nullptr : cs, rot_dims, interleaved);
            }
#pragma unroll
            for (int k = 0; k < LW_PIECES; ++k)
                if (i0 + 128 * k < heads * hq) store4(to[k], v[k]);
        }
    }
    // The sums of squares: a first pass over (the queries' latent, the cached row's), which the second finds in the cache.
    const int n_cq = in.cq != nullptr ? in.q_rank : 0, both = n_cq + (cached ? rank : 0);
    const float *cq_row = in.cq + (size_t)n * in.cq_ld, *dkv_row = in.dkv + (size_t)n * in.dkv_ld;
    float sq[LP_THREADS / 32] = {}, sc[LP_THREADS / 32] = {};
#pragma unroll 1
    for (int i0 = lane * 4; i0 < both; i0 += LP_THREADS * 4)
#pragma unroll
        for (int w = 0; w < LP_THREADS / 32; ++w) {
            const int i = i0 + w * 128;
            if (i >= both) continue;
            const float4 v = *reinterpret_cast<const float4*>(i < n_cq ? cq_row + i : dkv_row + i - n_cq);
            const float s = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w)));
            if (i < n_cq) sq[w] += s;
            else sc[w] += s;
        }
    // the cached row's latent, then the queries' own
    for (int part = 0; part < 2; ++part) {
        if (part == 0 ? !cached : in.cq == nullptr) continue;
        const float* row = part == 0 ? dkv_row : cq_row;
        const int count = part == 0 ? rank : in.q_rank;
        const float* w = part == 0 ? in.norm_w : in.cq_norm_w;
        T* dst = part == 0 ? cache + (size_t)slot * krow : cq_out + (size_t)n * in.q_rank;
        const float inv = 1.0f / sqrtf((part == 0 ? block_order_sum(sc, lane) : block_order_sum(sq, lane)) / (float)count + in.eps);
        for (int i0 = lane * 4; i0 < count; i0 += 128 * LW_PIECES) {
            float4 v[LW_PIECES], f[LW_PIECES];
#pragma unroll
            for (int k = 0; k < LW_PIECES; ++k)
                if (i0 + 128 * k < count) {
                    v[k] = *reinterpret_cast<const float4*>(row + i0 + 128 * k);
                    f[k] = *reinterpret_cast<const float4*>(w + i0 + 128 * k);
                }
#pragma unroll
            for (int k = 0; k < LW_PIECES; ++k)
                if (i0 + 128 * k < count)
                    store4(dst + i0 + 128 * k, make_float4(v[k].x * inv * f[k].x, v[k].y * inv * f[k].y, v[k].z * inv * f[k].z, v[k].w * inv * f[k].w));
        }
        if (part == 0)
            for (int d = lane * 4; d < rot_dim; d += 128) store4(dst + rank + d, turned4(row + rank, d, cs, rot_dims, interleaved));
    }
}

// out[n, h, o] = scale[n, h] * sum_k x[n, h, k] * W[h, o, k], k ascending per output.
// x rows: x + n * x_ld + h * x_hs; out rows: out + n * o_ld + h * o_hs.  Tiles of 32 tokens x 32
// outputs of one head; each of 256 threads owns a 2 x 2 patch.
constexpr int HB = 32, HK = 32;

template <typename T>
__global__ void __launch_bounds__(256)
headwise_linear_kernel(const T* __restrict__ x, long long x_ld, long long x_hs, const T* __restrict__ w,
                       T* __restrict__ out, long long o_ld, long long o_hs,
                       const float* __restrict__ scale, int N, int heads, int O, int K) {
    __shared__ float xs[HK][HB + 1];
    __shared__ float ws[HK][HB + 1];
    ie_pdl_trigger();
    ie_pdl_wait();
    int h = blockIdx.z, n0 = blockIdx.y * HB, o0 = blockIdx.x * HB;
    int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const T* wh = w + (size_t)h * O * K;
    float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    for (int k0 = 0; k0 < K; k0 += HK) {
        for (int i = tid; i < HB * HK; i += 256) {
            int r = i / HK, k = i - r * HK;
            float xv = 0.f, wv = 0.f;
            if (k0 + k < K) {
                if (n0 + r < N) xv = ie_load(x + (size_t)(n0 + r) * x_ld + (size_t)h * x_hs + k0 + k);
                if (o0 + r < O) wv = ie_load(wh + (size_t)(o0 + r) * K + k0 + k);
            }
            xs[k][r] = xv;
            ws[k][r] = wv;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < HK; ++k) {
            float a0 = xs[k][ty * 2], a1 = xs[k][ty * 2 + 1], b0 = ws[k][tx * 2], b1 = ws[k][tx * 2 + 1];
            acc[0][0] = fmaf(a0, b0, acc[0][0]); acc[0][1] = fmaf(a0, b1, acc[0][1]);
            acc[1][0] = fmaf(a1, b0, acc[1][0]); acc[1][1] = fmaf(a1, b1, acc[1][1]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        int n = n0 + ty * 2 + i;
        if (n >= N) continue;
        float f = scale ? scale[(size_t)n * heads + h] : 1.0f;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            int o = o0 + tx * 2 + j;
            if (o < O) ie_store(out + (size_t)n * o_ld + (size_t)h * o_hs + o, acc[i][j] * f);
        }
    }
}
// out[n, h, :] *= scale[n, h] (bfloat16 rows of `o` entries, rows n * o_ld + h * o_hs apart)
__global__ void scale_head_rows_kernel(__nv_bfloat16* __restrict__ out, long long o_ld, long long o_hs,
                                       const float* __restrict__ scale, int heads, int o) {
    ie_pdl_trigger();
    ie_pdl_wait();
    int n = blockIdx.x;
    for (int i = threadIdx.x; i < heads * o; i += blockDim.x) {
        int h = i / o, c = i - h * o;
        __nv_bfloat16* p = out + (size_t)n * o_ld + (size_t)h * o_hs + c;
        *p = __float2bfloat16_rn(__bfloat162float(*p) * scale[(size_t)n * heads + h]);
    }
}

// The same products on the tensor cores (bfloat16 weights, K a multiple of 16): W's rows are the
// instruction's 16 rows, tokens its columns.  XT float: x is the queries' 32-bit product (rounded to bfloat16
// here; in `x_parts` parts x_stride apart), and a head's last block turns the rotated part that follows x in its row
// (`rot`).  A block of four warps takes either 64 outputs, a warp each sixteen (SPLIT false), or sixteen
// outputs with K cut among its warps, whose sums are added in order (SPLIT true: long K, few outputs).
// grid: (output blocks, heads, blocks of 8 * NT tokens).
struct RotatedPart {
    const int* positions;
    const float* table;
    int rot_dims, table_rows, interleaved, rot_dim, at;  // the part starts `at` entries behind x; 0 entries: none
    int dst_at;                                           // ... and goes so many entries behind out
    int* err;
};

__device__ __forceinline__ void mma_m16n8k16(float* c, const unsigned* a, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <typename XT, int NT, bool SPLIT>
__global__ void __launch_bounds__(128)
headwise_mma_kernel(const XT* __restrict__ x, long long x_ld, long long x_hs, const __nv_bfloat16* __restrict__ w,
                    __nv_bfloat16* __restrict__ out, long long o_ld, long long o_hs, const float* __restrict__ scale,
                    RotatedPart rot, int x_parts, long long x_stride, bool fours, int N, int heads, int O, int K) {
    extern __shared__ __align__(16) unsigned char raw[];
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(raw);  // [8 * NT][K + 8]
    float* sums = reinterpret_cast<float*>(xs + 8 * NT * (K + 8));  // SPLIT: [4][16][8 * NT]
    ie_pdl_trigger();
    const int h = blockIdx.y, n0 = blockIdx.z * 8 * NT, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t4 = lane & 3, ld = K + 8;
    const int o0 = SPLIT ? blockIdx.x * 16 : (blockIdx.x * 4 + warp) * 16;
    const int steps = K / 16, k_begin = SPLIT ? warp * steps / 4 : 0, k_end = SPLIT ? (warp + 1) * steps / 4 : steps;
    // A thread's four consecutive entries of a row are the instruction's columns 2 t4, 2 t4 + 1 and 2 t4 + 8, 2 t4 + 9:
    // the same renaming of k for both operands.  The first steps' weights, which no kernel writes, are asked for
    // before the wait.
    const __nv_bfloat16* wa = w + ((size_t)h * O + (o0 + g < O ? o0 + g : 0)) * K + t4 * 4;
    const __nv_bfloat16* wb = w + ((size_t)h * O + (o0 + g + 8 < O ? o0 + g + 8 : 0)) * K + t4 * 4;
    constexpr int EARLY = 8;
    uint2 ra[EARLY], rb[EARLY];
#pragma unroll
    for (int i = 0; i < EARLY; ++i)
        if (k_begin + i < k_end) {
            ra[i] = *reinterpret_cast<const uint2*>(wa + (k_begin + i) * 16);
            rb[i] = *reinterpret_cast<const uint2*>(wb + (k_begin + i) * 16);
        }
    ie_pdl_wait();
    const int cnt = min(8 * NT, N - n0);
    if (rot.rot_dim > 0 && blockIdx.x + 1 == gridDim.x) {
        for (int i = tid; i < cnt * rot.rot_dim; i += 128) {
            int r = i / rot.rot_dim, d = i - r * rot.rot_dim, pos = rot.positions[n0 + r];
            bool turn = rot.table != nullptr && rot.rot_dims > 0;
            if (turn && (pos < 0 || pos >= rot.table_rows)) {
                if (d == 0) ie_report(rot.err, IE_ERR_POSITION, pos, n0 + r);
                turn = false;
            }
            const XT* p = x + (size_t)(n0 + r) * x_ld + (size_t)h * x_hs + rot.at;
            float v = 0.f;
            if constexpr (sizeof(XT) == 4)
                v = turned(Row{p, x_parts, (size_t)x_stride}, d, turn ? rot.table + (size_t)pos * rot.rot_dims : nullptr, rot.rot_dims, rot.interleaved);
            out[(size_t)(n0 + r) * o_ld + (size_t)h * o_hs + rot.dst_at + d] = __float2bfloat16_rn(v);
        }
        return;
    }
    for (int i = tid; i < 8 * NT * (K / 4); i += 128) {
        int r = i / (K / 4), c = (i - r * (K / 4)) * 4;
        uint2 v = make_uint2(0u, 0u);
        if (r < cnt) {
            const XT* p = x + (size_t)(n0 + r) * x_ld + (size_t)h * x_hs + c;
            if constexpr (sizeof(XT) == 4) {
                float4 f;
                if (fours) {
                    f = Row{p, x_parts, (size_t)x_stride}.four(0);
                } else {
                    const Row all{p, x_parts, (size_t)x_stride};
                    f = make_float4(all[0], all[1], all[2], all[3]);
                }
                __nv_bfloat162 lo = __floats2bfloat162_rn(f.x, f.y), hi = __floats2bfloat162_rn(f.z, f.w);
                v = make_uint2(*reinterpret_cast<unsigned*>(&lo), *reinterpret_cast<unsigned*>(&hi));
            } else if (fours) {
                v = *reinterpret_cast<const uint2*>(p);
            } else {
                __nv_bfloat162 lo = __halves2bfloat162(p[0], p[1]), hi = __halves2bfloat162(p[2], p[3]);
                v = make_uint2(*reinterpret_cast<unsigned*>(&lo), *reinterpret_cast<unsigned*>(&hi));
            }
        }
        *reinterpret_cast<uint2*>(xs + r * ld + c) = v;
    }
    __syncthreads();
    float c[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) c[t][0] = c[t][1] = c[t][2] = c[t][3] = 0.f;
    if (o0 < O) {
        auto step = [&](int kk, uint2 pa, uint2 pb) {
            unsigned a[4] = {pa.x, pb.x, pa.y, pb.y};
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                uint2 b = *reinterpret_cast<const uint2*>(xs + (t * 8 + g) * ld + kk * 16 + t4 * 4);
                mma_m16n8k16(c[t], a, b.x, b.y);
            }
        };
#pragma unroll
        for (int i = 0; i < EARLY; ++i)
            if (k_begin + i < k_end) step(k_begin + i, ra[i], rb[i]);
#pragma unroll 8
        for (int kk = k_begin + EARLY; kk < k_end; ++kk)
            step(kk, *reinterpret_cast<const uint2*>(wa + kk * 16), *reinterpret_cast<const uint2*>(wb + kk * 16));
    }
    if constexpr (SPLIT) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            float* dst = sums + (warp * 16 + g) * 8 * NT + t * 8 + t4 * 2;
            dst[0] = c[t][0]; dst[1] = c[t][1];
            dst[64 * NT] = c[t][2]; dst[64 * NT + 1] = c[t][3];
        }
        __syncthreads();
        for (int i = tid; i < 16 * 8 * NT; i += 128) {
            int o = i % 16, r = i / 16, at = o * 8 * NT + r;
            if (r >= cnt || o0 + o >= O) continue;
            float v = ((sums[at] + sums[128 * NT + at]) + sums[256 * NT + at]) + sums[384 * NT + at];
            if (scale) v *= scale[(size_t)(n0 + r) * heads + h];
            out[(size_t)(n0 + r) * o_ld + (size_t)h * o_hs + o0 + o] = __float2bfloat16_rn(v);
        }
    } else {
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                int o = o0 + g + (e >> 1) * 8, r = t * 8 + t4 * 2 + (e & 1);
                if (o >= O || r >= cnt) continue;
                float v = c[t][e];
                if (scale) v *= scale[(size_t)(n0 + r) * heads + h];
                out[(size_t)(n0 + r) * o_ld + (size_t)h * o_hs + o] = __float2bfloat16_rn(v);
            }
    }
}

template <typename XT, int NT, bool SPLIT>
int launch_headwise_mma(const void* x, long long x_ld, long long x_hs, const void* w, void* out, long long o_ld,
                        long long o_hs, const float* scale, RotatedPart rot, int x_parts, long long x_stride, int N,
                        int heads, int O, int K, cudaStream_t s) {
    size_t smem = (size_t)8 * NT * (K + 8) * 2 + (SPLIT ? (size_t)4 * 16 * 8 * NT * 4 : 0);
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, headwise_mma_kernel<XT, NT, SPLIT>, 96 * 1024);
    if (e != cudaSuccess) return (int)e;
    const bool fours = x_ld % 4 == 0 && x_hs % 4 == 0 && x_stride % 4 == 0 && reinterpret_cast<uintptr_t>(x) % (4 * sizeof(XT)) == 0;
    dim3 grid((SPLIT ? (O + 15) / 16 : (O + 63) / 64) + (rot.rot_dim > 0 ? 1 : 0), heads, (N + 8 * NT - 1) / (8 * NT));
    return ie_launch(headwise_mma_kernel<XT, NT, SPLIT>, grid, dim3(128), smem, s, (const XT*)x, x_ld, x_hs,
                     (const __nv_bfloat16*)w, (__nv_bfloat16*)out, o_ld, o_hs, scale, rot, x_parts, x_stride, fours, N, heads, O, K);
}

template <typename XT>
int pick_headwise_mma(const void* x, long long x_ld, long long x_hs, const void* w, void* out, long long o_ld,
                      long long o_hs, const float* scale, RotatedPart rot, int x_parts, long long x_stride, int N,
                        int heads, int O, int K, cudaStream_t s) {
#define IE_HM_ARGS x, x_ld, x_hs, w, out, o_ld, o_hs, scale, rot, x_parts, x_stride, N, heads, O, K, s
    // (the cut must not change with the number of tokens: a token's sums depend on the sizes alone)
    bool split = K >= 256;
    if (N <= 8) return split ? launch_headwise_mma<XT, 1, true>(IE_HM_ARGS) : launch_headwise_mma<XT, 1, false>(IE_HM_ARGS);
    return split ? launch_headwise_mma<XT, 4, true>(IE_HM_ARGS) : launch_headwise_mma<XT, 4, false>(IE_HM_ARGS);
#undef IE_HM_ARGS
}

// A warp per row: the cached rows of the step's requests, whole contexts one after the other, into an array without gaps.
__global__ void __launch_bounds__(256)
gather_context_rows_kernel(const uint4* __restrict__ cache, const int* __restrict__ tables, int table_width,
                           const int* __restrict__ ctx_lens, int num_seqs, int total, int pieces, int page_shift, int total_pages,
                           uint4* __restrict__ out, int* err) {
    ie_pdl_trigger();
    ie_pdl_wait();
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= total) return;
    int seq = 0, pos = row;
    while (seq < num_seqs && pos >= ctx_lens[seq]) pos -= ctx_lens[seq++];
    if (seq >= num_seqs) return;
    const int page = tables[(size_t)seq * table_width + (pos >> page_shift)];
    if (page < 0 || page >= total_pages) {
        if (lane == 0) ie_report(err, page < 0 ? IE_ERR_TABLE : IE_ERR_PAGE, page, row);
        return;
    }
    const uint4* src = cache + (((size_t)page << page_shift) + (pos & ((1 << page_shift) - 1))) * pieces;
    for (int i = lane; i < pieces; i += 32) out[(size_t)row * pieces + i] = src[i];
}
}  // namespace

IE_API int ie_scale_head_rows(void* out, long long o_ld, long long o_hs, const float* scale, int N, int heads, int o,
                              void* stream) {
    if (N <= 0) return 0;
    return ie_launch(scale_head_rows_kernel, dim3(N), dim3(256), 0, (cudaStream_t)stream, (__nv_bfloat16*)out, o_ld, o_hs,
                     scale, heads, o);
}

IE_API int ie_latent_prep(const float* q, int q_ld, const float* gate_pre, int gate_ld, const float* dkv, int dkv_ld,
                          const float* cq, int cq_ld, int q_rank, int parts, long long part_stride, const float* norm_w, const float* cq_norm_w, float eps,
                          const int* positions, const float* table, int rot_dims, int table_rows, int interleaved,
                          void* q_plain, void* q_abs, float* gate, void* cq_out, void* cache, int dtype,
                          const int* slot_mapping, int num_tokens, int heads, int dim, int rot_dim, int rank,
                          int total_slots, int* err, void* stream) {
    if (num_tokens <= 0) return 0;
    if (rot_dims < 0 || rot_dims % 2 || rot_dims > rot_dim) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    if (parts < 1) return (int)cudaErrorInvalidValue;
    LatentIn in{q, q_ld, gate_pre, gate_ld, dkv, dkv_ld, cq, cq_ld, q_rank, parts, (size_t)part_stride, norm_w, cq_norm_w, eps, false, false};
    in.fours = q_rank % 4 == 0 && rank % 4 == 0 && rot_dim % 4 == 0 && cq_ld % 4 == 0 && dkv_ld % 4 == 0 && part_stride % 4 == 0 &&
               ((reinterpret_cast<uintptr_t>(cq) | reinterpret_cast<uintptr_t>(dkv)) % 16 == 0);
    in.all_fours = parts == 1 && in.fours && dim % 4 == 0 && rot_dims % (interleaved ? 4 : 8) == 0 && q_ld % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(q_plain) | reinterpret_cast<uintptr_t>(q_abs) |
                     reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(norm_w) | reinterpret_cast<uintptr_t>(cq_norm_w) |
                     reinterpret_cast<uintptr_t>(cq_out) | reinterpret_cast<uintptr_t>(cache)) % 16 == 0);
    size_t smem = ((cq ? q_rank : 0) + (dkv ? rank + rot_dim : 0)) * sizeof(float);
    if (smem > 40 * 1024) return (int)cudaErrorInvalidValue;
    // (from four tokens an SM on: fewer are done sooner with a block each)
    if (in.all_fours && num_tokens >= 4 * ie_sm_count()) {
        const dim3 grid((num_tokens + LW_WARPS - 1) / LW_WARPS), block(LW_WARPS * 32);
        if (dtype == IE_BF16)
            return ie_launch(latent_prep_warp_kernel<__nv_bfloat16>, grid, block, 0, s, in, positions, table, rot_dims, table_rows, interleaved,
                             (__nv_bfloat16*)q_plain, (__nv_bfloat16*)q_abs, gate, (__nv_bfloat16*)cq_out, (__nv_bfloat16*)cache,
                             slot_mapping, num_tokens, heads, dim, rot_dim, rank, total_slots, err);
        return ie_launch(latent_prep_warp_kernel<float>, grid, block, 0, s, in, positions, table, rot_dims, table_rows, interleaved,
                         (float*)q_plain, (float*)q_abs, gate, (float*)cq_out, (float*)cache, slot_mapping, num_tokens, heads, dim, rot_dim,
                         rank, total_slots, err);
    }
    if (dtype == IE_BF16)
        return ie_launch(latent_prep_kernel<__nv_bfloat16>, dim3(num_tokens), dim3(LP_THREADS), smem, s, in, positions, table,
                         rot_dims, table_rows, interleaved, (__nv_bfloat16*)q_plain, (__nv_bfloat16*)q_abs, gate,
                         (__nv_bfloat16*)cq_out, (__nv_bfloat16*)cache, slot_mapping, heads, dim, rot_dim, rank,
                         total_slots, err);
    return ie_launch(latent_prep_kernel<float>, dim3(num_tokens), dim3(LP_THREADS), smem, s, in, positions, table, rot_dims,
                     table_rows, interleaved, (float*)q_plain, (float*)q_abs, gate, (float*)cq_out, (float*)cache,
                     slot_mapping, heads, dim, rot_dim, rank, total_slots, err);
}

// Whether headwise_mma takes this inner size (else headwise_linear runs).
IE_API int ie_headwise_mma_ok(int K) { return K % 16 == 0 && K >= 16 && K <= 1024; }

// x: bfloat16, or 32-bit (x_f32) with a rotated part of rot_dim entries that starts `rot_at` entries behind x.
IE_API int ie_headwise_mma(const void* x, int x_f32, long long x_ld, long long x_hs, const void* w, void* out,
                           long long o_ld, long long o_hs, const float* scale, int N, int heads, int O, int K,
                           int x_parts, long long x_stride, const int* positions, const float* table, int rot_dims,
                           int table_rows, int interleaved, int rot_dim, int rot_at, int rot_dst, int* err, void* stream) {
    if (N <= 0 || heads <= 0 || O <= 0) return 0;
    if (!ie_headwise_mma_ok(K) || x_parts < 1 || (rot_dim > 0 && (!x_f32 || positions == nullptr)) || rot_dims < 0 || rot_dims % 2 ||
        rot_dims > rot_dim || reinterpret_cast<uintptr_t>(w) % 8)
        return (int)cudaErrorInvalidValue;
    RotatedPart rot{positions, table, rot_dims, table_rows, interleaved, rot_dim, rot_at, rot_dst, err};
    cudaStream_t s = (cudaStream_t)stream;
    if (x_f32) return pick_headwise_mma<float>(x, x_ld, x_hs, w, out, o_ld, o_hs, scale, rot, x_parts, x_stride, N, heads, O, K, s);
    return pick_headwise_mma<__nv_bfloat16>(x, x_ld, x_hs, w, out, o_ld, o_hs, scale, rot, x_parts, x_stride, N, heads, O, K, s);
}

IE_API int ie_headwise_linear(const void* x, long long x_ld, long long x_hs, const void* w, void* out,
                              long long o_ld, long long o_hs, const float* scale, int dtype, int N, int heads,
                              int O, int K, void* stream) {
    if (N <= 0 || heads <= 0 || O <= 0) return 0;
    dim3 grid((O + HB - 1) / HB, (N + HB - 1) / HB, heads);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == IE_BF16)
        return ie_launch(headwise_linear_kernel<__nv_bfloat16>, grid, dim3(256), 0, s, (const __nv_bfloat16*)x, x_ld,
                         x_hs, (const __nv_bfloat16*)w, (__nv_bfloat16*)out, o_ld, o_hs, scale, N, heads, O, K);
    return ie_launch(headwise_linear_kernel<float>, grid, dim3(256), 0, s, (const float*)x, x_ld, x_hs,
                     (const float*)w, (float*)out, o_ld, o_hs, scale, N, heads, O, K);
}

// cache: bfloat16 [pages, page_size, row], row a multiple of 8; out: [total, row], the requests' contexts one after the other.
IE_API int ie_gather_context_rows(const void* cache, const int* tables, int table_width, const int* ctx_lens, int num_seqs, int total,
                                  int row, int page_size, int total_pages, void* out, int* err, void* stream) {
    if (total <= 0) return 0;
    if (row % 8 || page_size < 1 || (page_size & (page_size - 1)) || (((uintptr_t)cache | (uintptr_t)out) & 15)) return (int)cudaErrorInvalidValue;
    int shift = 0;
    while ((1 << shift) < page_size) ++shift;
    return ie_launch(gather_context_rows_kernel, dim3((total + 7) / 8), dim3(256), 0, (cudaStream_t)stream, (const uint4*)cache, tables,
                     table_width, ctx_lens, num_seqs, total, row / 8, shift, total_pages, (uint4*)out, err);
}
