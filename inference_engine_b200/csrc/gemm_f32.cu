// True 32-bit matrix product:  C[M, N] = A[M, K] * W[N, K]^T, the matrix product of the engine's 32-bit path.
//
// Every output element is the same sums in the same order, whatever the tile: the result of a row does not depend on how many other rows the
// step has, on where the row sits in the batch or on the tile it falls into.  That makes 32-bit logits identical however the tokens were cut
// into steps.  Which sums depends on K alone.  Below MMA_K: one chain of fused multiply-adds over k = 0 .. K-1 on the CUDA cores.
// From there on: products put together on the tensor cores (from three products of parts of 11 bits; their TF32 mode by itself drops mantissa
// bits), summed by sixteens, those in four chains of 32-bit adders.  The shorter chains leave less error than one long one: against 64 bits, as
// a part of the result, one chain / so, for normal numbers 1.4e-7 / 1.1e-7 at K = 64, 2.9e-7 / 1.2e-7 at 256, 5.7e-7 / 1.3e-7 at 1,024 and
// 11.5e-7 / 1.8e-7 at 4,096; for terms that grow a hundredfold along k, where a chain is best, 1.0e-7 / 1.1e-7 at 128 and 1.3e-7 / 1.1e-7
// at 256.  From 256 on it was lower for those, for positive, shrinking and cancelling terms and for ones of very different sizes.
// The reference's 32-bit path is cuBLAS with TF32 off (PyTorch's default).
#include "split32.cuh"

namespace {
constexpr int BK = 16, TN = 4, BN = 64, THREADS = 128, AHEAD = 4, MMA_K = 256;

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
// the same chain over k.  (By 1,024 of k, which the other kernel takes by now, us, with tiles of 64 x 64, with these and one tile ahead, and with four: 8 rows by
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

// ---- the same on the tensor cores ----

// One chain of multiply-adds: for what is no finite number, which parts that are subtracted from one another do not keep as it is.
__device__ __noinline__ float one_chain(const float* __restrict__ a, const float* __restrict__ w, int K) {
    float s = 0.f;
#pragma unroll 1
    for (int k = 0; k < K; ++k) s = fmaf(a[k], w[k], s);
    return s;
}
// A block: BM x BN in tiles of WM x 32, four warps a tile: of every 64 of k a warp takes its own 16, and the four sums are added at the end.
// So an output is the same sums in the same order whatever the block, and a short step has warps enough although the tiles are
// large: the operands are taken apart by every warp that reads them, which with tiles of 16 x 16 is more work than the products.
// A stage is 64 of k in four slabs of 16, STAGES of them.  A row of a slab is 64 bytes, of which a lane takes 16, four k: the lanes that are
// served together meet in no bank, and one load feeds two of the tensor cores' eights.
// VEC: rows of whole 16-byte pieces, aligned.
// What bounds it: the products and what takes the operands apart, 10 clocks of a scheduler for a product that takes 8, and, of short steps, the way
// to the first stage and back.  By 1,024 of k, us, with the kernel above / so: 8 rows by 4,096 29 / 10, 377 by 1,536 44 / 27, 377 by 1,024
// 43 / 23, 2,048 by 2,048 203 / 158; 160 by 2,048 of 8,192 of k 330 / 145.  (Three stages, so that four blocks of 32 x 32 fit an SM; with four
// stages and three blocks 29, 23, 164 and 143.)  (A warp the whole of k of its tile: 31, 25 and 187 for
// 377 by 1,536, by 1,024 and 2,048 by 2,048 with tiles of 16 x 16 a warp, 29, 29 and 148 with 32 x 32; 64 x 64 a block of 16 warps 29, 29
// and 180.)
template <int BM, int BN, int WM, int STAGES, bool VEC>
__global__ void __launch_bounds__(BM / WM * BN / 32 * 128, BM == 32 ? 4 : 1)
gemm_f32_mma_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K) {
    constexpr int WN = 32, TILES = BM / WM * BN / WN, T = TILES * 128, ROWS = BM + BN, STEP = 64, SLAB = ROWS * 16, MT = WM / 16, NT = WN / 8;
    constexpr int PASS = T / 16;  // rows that the block's threads fetch at once
    static_assert(ROWS % PASS == 0 && BM % PASS == 0 && TILES * 4 * 32 * MT * NT * 4 <= STAGES * 4 * SLAB, "");
    extern __shared__ __align__(16) float sm[];
    ie_pdl_trigger();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, part = warp & 3, tile = warp >> 2;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, wm = tile / (BN / WN) * WM, wn = tile % (BN / WN) * WN;
    const int piece = tid & 15, first = tid >> 4;  // the thread's four k of a stage, and its rows: every PASS-th
    auto fetch = [&](int k0, int stage) {
        const int k = k0 + 4 * piece;
        unsigned dst = (unsigned)__cvta_generic_to_shared(sm + (4 * stage + (piece >> 2)) * SLAB + first * 16 + (piece & 3) * 4);
#pragma unroll
        for (int i = 0; i < ROWS / PASS; ++i, dst += PASS * 64) {
            const int row = first + PASS * i;
            const bool is_a = i < BM / PASS;
            const int at = is_a ? m0 + row : n0 + row - BM;
            const bool there = at < (is_a ? M : N);
            const float* src = (is_a ? A : W) + (there ? (size_t)at * K : 0);
            if (VEC) {
                const bool some = there && k < K;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src + (some ? k : 0)), "r"(some ? 16 : 0) : "memory");
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const bool some = there && k + e < K;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * e), "l"(src + (some ? k + e : 0)), "r"(some ? 4 : 0) : "memory");
                }
            }
        }
    };
    const int steps = (K + STEP - 1) / STEP;
    ie_pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) fetch(s * STEP, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[MT][NT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;
    int stage = 0, next = STAGES - 1;
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();  // the stage is here, and nobody reads the one that is fetched next
        if (s + STAGES - 1 < steps) fetch((s + STAGES - 1) * STEP, next);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* slab = sm + (4 * stage + part) * SLAB + 4 * t;
        Two a[MT][2][4];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const float4 x = *reinterpret_cast<const float4*>(slab + (wm + 16 * m + g) * 16);
            const float4 y = *reinterpret_cast<const float4*>(slab + (wm + 16 * m + 8 + g) * 16);
            a[m][0][0] = apart(x.x); a[m][0][1] = apart(y.x); a[m][0][2] = apart(x.y); a[m][0][3] = apart(y.y);
            a[m][1][0] = apart(x.z); a[m][1][1] = apart(y.z); a[m][1][2] = apart(x.w); a[m][1][3] = apart(y.w);
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const float4 z = *reinterpret_cast<const float4*>(slab + (BM + wn + 8 * n + g) * 16);
            Two b[2][2];
            two(z.x, z.y, b[0][0], b[0][1]);
            two(z.z, z.w, b[1][0], b[1][1]);
            float c[MT][4];
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int m = 0; m < MT; ++m) mma6_part(c[m], i, a[m], b);
#pragma unroll
            for (int m = 0; m < MT; ++m) add_to(acc[m][n], c[m]);
        }
        stage = stage + 1 == STAGES ? 0 : stage + 1;
        next = next + 1 == STAGES ? 0 : next + 1;
    }
    // the four warps' sums: each adds up a quarter of the tile
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    constexpr int EACH = MT * NT / 4;
    float4* sums = reinterpret_cast<float4*>(sm) + tile * 4 * MT * NT * 32 + lane;  // [part][8 x 16 tiles][lane]
#pragma unroll
    for (int i = 0; i < MT * NT; ++i) {
        const float* v = acc[i / NT][i % NT];
        sums[(part * MT * NT + i) * 32] = make_float4(v[0], v[1], v[2], v[3]);
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < EACH; ++e) {
        const int i = part * EACH + e;
        float v[4][4];
#pragma unroll
        for (int p = 0; p < 4; ++p) *reinterpret_cast<float4*>(v[p]) = sums[(p * MT * NT + i) * 32];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int gm = m0 + wm + 16 * (i / NT) + g + (r >> 1) * 8, gn = n0 + wn + 8 * (i % NT) + 2 * t + (r & 1);
            if (gm >= M || gn >= N) continue;
            float x = (v[0][r] + v[1][r]) + (v[2][r] + v[3][r]);
            if (!isfinite(x)) x = one_chain(A + (size_t)gm * K, W + (size_t)gn * K, K);
            C[(size_t)gm * N + gn] = x;
        }
    }
}

template <int BM, int BN, int WM, int STAGES>
cudaError_t launch_mma(const float* A, const float* W, float* C, int M, int N, int K, bool vec, cudaStream_t s) {
    constexpr size_t smem = (size_t)STAGES * (BM + BN) * 64 * sizeof(float);
    static IePerDevice allowed_vec, allowed;
    auto kernel = vec ? gemm_f32_mma_kernel<BM, BN, WM, STAGES, true> : gemm_f32_mma_kernel<BM, BN, WM, STAGES, false>;
    cudaError_t e = ie_allow_smem(vec ? allowed_vec : allowed, kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<dim3((N + BN - 1) / BN, (M + BM - 1) / BM), dim3(BM / WM * BN / 32 * 128), smem, s>>>(A, W, C, M, N, K);
    return cudaSuccess;
}
}  // namespace

IE_API int ie_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    const bool vec = K % 4 == 0 && !(((size_t)A | (size_t)W) & 15);
    if (K >= MMA_K) {
        // (16 rows a block for a few rows, or where blocks of 32 rows would leave half of the SMs idle: 64 rows by 1,024 10 us against 12, 128 by
        // 3,072 27 against 23; an output is the same either way)
        const long long blocks = (long long)((M + 31) / 32) * ((N + 31) / 32);
        const bool few = M <= 16 || 2 * blocks <= ie_sm_count();
        cudaError_t e = few ? launch_mma<16, 32, 16, 5>(A, W, C, M, N, K, vec, (cudaStream_t)stream)
                            : launch_mma<32, 32, 32, 3>(A, W, C, M, N, K, vec, (cudaStream_t)stream);
        return e != cudaSuccess ? (int)e : IE_LAUNCH_CHECK();
    }
    const int across = (N + BN - 1) / BN;
    // (64 rows a block once such blocks are two to an SM; below that 32, so that more SMs have one)
    const bool large = (long long)((M + 63) / 64) * across >= 2ll * ie_sm_count();
    const dim3 grid(across, large ? (M + 63) / 64 : (M + 31) / 32);
    auto kernel = large ? (vec ? gemm_f32_kernel<64, true> : gemm_f32_kernel<64, false>) : (vec ? gemm_f32_kernel<32, true> : gemm_f32_kernel<32, false>);
    // A plain launch: blocks that start while the kernel before still runs go where there is room, four on one SM and none on another.
    kernel<<<grid, dim3(THREADS), 0, (cudaStream_t)stream>>>(A, W, C, M, N, K);
    return IE_LAUNCH_CHECK();
}
