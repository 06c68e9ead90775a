// True 32-bit matrix product on the CUDA cores:  C[M, N] = A[M, K] * W[N, K]^T.
//
// No tensor-core mode is involved (tcgen05 has no 32-bit input kind and TF32 drops mantissa
// bits), so this is the matrix product of the engine's 32-bit path.  Every output element is
// one chain of fused multiply-adds over k = 0 .. K-1 in increasing order: the result of a row
// does not depend on how many other rows the step has, on where the row sits in the batch or
// on the tile it falls into.  That makes 32-bit logits identical however the tokens were cut
// into steps.  The reference's 32-bit path is cuBLAS with TF32 off (PyTorch's default).
#include "common.cuh"

namespace {
constexpr int BK = 16, TN = 4, BN = 64, THREADS = 128, AHEAD = 4;

// Two multiply-adds in one instruction, each rounded as one by itself: the kernel is bound by the instructions it issues.
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long twice(float x) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}

// A block: BM rows x 64 columns, 8 x 16 threads; a thread TM = BM / 8 rows (in pairs) x 4 columns.  The next four times 16 of k are fetched
// into registers while these are worked on: 16 of k are some 600 clocks of work, less than a trip to memory takes.  Whatever the tile, an output is
// the same chain over k.  (By 1,024 of k, us, with the tiles of 64 x 64 that were here first, with these and one tile ahead, and with four: 8 rows by
// 4,096 53, 33 and 29, 377 by 1,536 55, 52 and 44, 2,048 by 2,048 258, 208 and 203.  The instructions issued bound the larger ones.)
// VEC: rows of whole 16-byte pieces, aligned.
template <int BM, bool VEC>
__global__ void __launch_bounds__(THREADS)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K) {
    constexpr int TM = BM / 8, A_LOADS = BM * BK / 4 / THREADS, W_LOADS = BN * BK / 4 / THREADS;
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Ws[2][BK][BN + 4];
    ie_pdl_trigger();
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16, m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    // four consecutive k of one row
    auto fetch = [&](const float* __restrict__ X, int row, int rows, int k) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* p = X + (size_t)row * K + k;
        if (row >= rows || k >= K) return v;
        if (VEC) return *reinterpret_cast<const float4*>(p);
        v.x = p[0];
        if (k + 1 < K) v.y = p[1];
        if (k + 2 < K) v.z = p[2];
        if (k + 3 < K) v.w = p[3];
        return v;
    };
    float4 a[AHEAD][A_LOADS], w[AHEAD][W_LOADS];
    auto fetch_a = [&](int k0, int set) {
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) a[set][i] = fetch(A, m0 + (tid + i * THREADS) / 4, M, k0 + (tid % 4) * 4);
    };
    auto fetch_w = [&](int k0, int set) {
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) w[set][i] = fetch(W, n0 + (tid + i * THREADS) / 4, N, k0 + (tid % 4) * 4);
    };
    auto keep_tile = [&](int b, int set) {
        const int k = (tid % 4) * 4;
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            const int r = (tid + i * THREADS) / 4;
            As[b][k][r] = a[set][i].x; As[b][k + 1][r] = a[set][i].y; As[b][k + 2][r] = a[set][i].z; As[b][k + 3][r] = a[set][i].w;
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            const int r = (tid + i * THREADS) / 4;
            Ws[b][k][r] = w[set][i].x; Ws[b][k + 1][r] = w[set][i].y; Ws[b][k + 2][r] = w[set][i].z; Ws[b][k + 3][r] = w[set][i].w;
        }
    };
    unsigned long long acc[TM / 2][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
#pragma unroll
    for (int set = 0; set < AHEAD; ++set) fetch_w(set * BK, set);  // (weights: nothing that the kernel before writes)
    ie_pdl_wait();
#pragma unroll
    for (int set = 0; set < AHEAD; ++set) fetch_a(set * BK, set);
    keep_tile(0, 0);
    __syncthreads();
    for (int k1 = 0; k1 < K; k1 += AHEAD * BK)
#pragma unroll
    for (int set = 0; set < AHEAD; ++set) {
        const int k0 = k1 + set * BK, b = set & 1;
        if (k0 >= K) break;
        const bool more = k0 + BK < K;
        fetch_a(k0 + AHEAD * BK, set);  // (beyond K: zeros, nothing is read)
        fetch_w(k0 + AHEAD * BK, set);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const float4 wv = *reinterpret_cast<const float4*>(&Ws[b][k][tx * TN]);
            const unsigned long long w2[TN] = {twice(wv.x), twice(wv.y), twice(wv.z), twice(wv.w)};
#pragma unroll
            for (int i = 0; i < TM / 4; ++i) {
                const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(&As[b][k][ty * TM + 4 * i]);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[2 * i][j] = fma2(av.x, w2[j], acc[2 * i][j]);
                    acc[2 * i + 1][j] = fma2(av.y, w2[j], acc[2 * i + 1][j]);
                }
            }
        }
        if (more) keep_tile(b ^ 1, (set + 1) % AHEAD);  // (everyone is done with that buffer since the last barrier)
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            const unsigned long long pair = acc[i / 2][j];
            if (gn < N) C[(size_t)gm * N + gn] = __uint_as_float(i & 1 ? (unsigned)(pair >> 32) : (unsigned)pair);
        }
    }
}
}  // namespace

IE_API int ie_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const int across = (N + BN - 1) / BN;
    // (64 rows a block once such blocks are two to an SM; below that 32, so that more SMs have one)
    const bool large = (long long)((M + 63) / 64) * across >= 2ll * ie_sm_count(), vec = K % 4 == 0 && !(((size_t)A | (size_t)W) & 15);
    const dim3 grid(across, large ? (M + 63) / 64 : (M + 31) / 32);
    auto kernel = large ? (vec ? gemm_f32_kernel<64, true> : gemm_f32_kernel<64, false>) : (vec ? gemm_f32_kernel<32, true> : gemm_f32_kernel<32, false>);
    // A plain launch: blocks that start while the kernel before still runs go where there is room, four on one SM and none on another.
    kernel<<<grid, dim3(THREADS), 0, (cudaStream_t)stream>>>(A, W, C, M, N, K);
    return IE_LAUNCH_CHECK();
}
