// Recurrences of matrix states over long portions, 64 tokens at a time, in 32-bit throughout.
//
//   S_t = diag(a_t) S_(t-1) + w_t u_t^T,   o_t = S_t^T q_t          (linear attention with decays)
//   u_t = beta_t (v_t - (diag(a_t) S_(t-1))^T k_t),  w_t = k_t       (the gated delta rule)
//
// Token by token a state entry waits for its own last value and a portion's 128 blocks keep a warp per scheduler busy
// every few clocks.  Cut into chunks of 64 the same sums become small products.  With D(i, j) = a_(j+1) ... a_i per channel, S0 the state
// before the chunk and p_i = a_1 ... a_i:
//   o_i = (p_i q_i)^T S0 + sum_(j <= i) A(i, j) u_j,   A(i, j) = sum_d q_i D(i, j) w_j
//   S_after = diag(p_last) S0 + sum_j (D(last, j) w_j) u_j^T
// No decay is ever divided by another or turned into a logarithm (a decay may be 0): D is a product of running products
// inside groups of 16 tokens (from the group's start to i, from j to its group's end) and of whole groups between; inside one group
// it is multiplied up pair by pair.
//
//  * chunk_state: what a chunk by itself adds to the state, and its decay (a block per chunk and head).
//  * chunk_scan: the state runs through a request's chunks and is left, before each chunk, in that chunk's place.
//  * chunk_out: the outputs (a block per chunk and head: 64 x 64 scores, then 64 x dim x cols and 64 x 64 x cols).
// The delta rule's u depend on the state, (I + diag(beta) L) u = diag(beta) (v - (p k)^T S0), L(i, j) = k_i D(i, j) k_j below the
// diagonal:
//  * delta_solve: both right-hand sides by forward substitution in blocks of 16: U = X v, W = X (p k).
//  * delta_chain: u = U - W S0 and the state after, chunk after chunk; columns of S do not interact, so a block takes 16
//    columns of a head and keeps them in registers; the next chunk's W and decayed keys are on their way meanwhile.
//  * chunk_out with those u.
//
// What bounds it: the multiply-adds, 40 thousand per token and head of 128 x 128, and what brings their operands from shared memory.  A
// state in 32 bits must not lose precision, so the products are 32-bit ones, put together from three of the tensor cores' on parts
// of 11 bits (below); the FMA pipe alone, two operands from shared memory to every few multiply-adds, took longer.  2,048 tokens, 16 heads of
// 128 x 128, us with FMAs / so: outputs 79 / 66 (delta rule 81 / 70), solve 75 / 54, chain 111 / 84; all
// together 142 / 122 and 270 / 214.  (Outputs 61 since their scores do not wait for the states.)  Errors against 64 bits, over keys of 64 and 128, as parts of the results: outputs 1.4e-7 / 1.3e-7, of the delta rule 2.6e-7 /
// 2.1e-7, its states 1.9e-7 / 1.8e-7.
#include "split32.cuh"
#include <float.h>

namespace {

constexpr int CHUNK = 64, GROUP = 16, THREADS = 256;

// Which request and which of its chunks the block's chunk number means; false: there are fewer chunks.
__device__ __forceinline__ bool find_chunk(const int* cu_q, int num_seqs, int number, int& seq, int& chunk) {
    for (seq = 0; seq < num_seqs; ++seq) {
        int n = (cu_q[seq + 1] - cu_q[seq] + CHUNK - 1) / CHUNK;
        if (number < n) { chunk = number; return true; }
        number -= n;
    }
    return false;
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool there) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}

// ROWS rows of `dim` entries `ld` apart into rows LD apart, zeros beyond the chunk's rows and beyond dim.
template <int ROWS, int DIM, int LD>
__device__ __forceinline__ void fetch_rows(float* dst, const float* src, size_t ld, int cnt, int dim) {
#pragma unroll
    for (int i = threadIdx.x; i < ROWS * DIM / 4; i += THREADS) {
        int row = i / (DIM / 4), piece = i % (DIM / 4);
        bool there = row < cnt && piece * 4 < dim;
        cp16(dst + row * LD + piece * 4, there ? src + row * ld + piece * 4 : src, there);
    }
}

__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }

// Rows that the tensor cores read along k lie DIM + 8 apart, rows that they read across it so many columns + 4: no two lanes that are
// served together then meet in a bank.
template <int DIM> constexpr int along() { return DIM + 8; }

// N tiles of 16 x 8 side by side: acc += rows a (k along) times rows b (k along), K of them.  `of_a`, `of_b`: what a value pair is multiplied by (k).
template <int K, int N, typename FA, typename FB>
__device__ __forceinline__ void tile_product(float (&acc)[N][4], const float* a, int a_ld, const float* b, int b_ld, FA of_a, FB of_b) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t2 = (lane & 3) * 2;
    const float *a0 = a + g * a_ld + t2, *a1 = a0 + 8 * a_ld, *bp = b + g * b_ld + t2;
#pragma unroll 4
    for (int k = 0; k < K; k += 16) {
        Two av[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 x = of_a(ld2(a0 + k + 8 * h), 0, k + 8 * h + t2), y = of_a(ld2(a1 + k + 8 * h), 1, k + 8 * h + t2);
            av[h][0] = apart(x.x);
            av[h][1] = apart(y.x);
            av[h][2] = apart(x.y);
            av[h][3] = apart(y.y);
        }
#pragma unroll
        for (int n = 0; n < N; ++n) {
            Two bv[2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 z = of_b(ld2(bp + 8 * n * b_ld + k + 8 * h), k + 8 * h + t2);
                two(z.x, z.y, bv[h][0], bv[h][1]);
            }
            float c[4];
            mma6(c, av, bv);
            add_to(acc[n], c);
        }
    }
}

// The scores of a chunk, A(i, j) = sum_d q_i D(i, j) w_j for j <= i, at A[i * A_LD + j] (TRANS: A[j * A_LD + i]); nothing above the diagonal.
// Left behind: qs: [64][DIM + 8], q_i times the decays from its group's start to i; ws: the same shape, w_j times the decays from j + 1 to its
// group's end; total: [4][DIM], the groups' whole decays; ahead: [4][DIM], those of all groups before.  quad: [16][DIM], scratch.
// Four neighbouring tokens' pairs are multiplied up where they are read; every other pair's decay is a product of running products: inside
// the four, of whole fours between (in groups of 16), of whole groups between.  16 x 16 blocks then are products along d for the
// tensor cores, also the one on the diagonal (of which a quarter is wanted).  (16 tokens' pairs multiplied up and the blocks between
// as multiply-adds, all from shared memory: 64 of the delta rule's 73 us for its solves of 2,048 tokens and 16 heads of 128 x 128.)
template <int DIM, bool TRANS>
struct Scores {
    static constexpr int LD = along<DIM>(), A_LD = CHUNK + 8;
    static __device__ __forceinline__ int at(int i, int j) { return TRANS ? j * A_LD + i : i * A_LD + j; }

    // q, w, a of a row's four entries (zeros and ones beyond the chunk): functions of (row, first entry)
    template <typename Q, typename W, typename D>
    static __device__ __forceinline__ void run(float* qs, float* ws, float* quad, float* total, float* ahead, float* A, Q q_of, W w_of, D a_of) {
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        constexpr int LANES = DIM / 4, AT_ONCE = THREADS / LANES;  // 32 lanes, 8 fours at once; or 16, 16
        {
            const int sub = tid % LANES, d = sub * 4;
#pragma unroll 1
            for (int b = tid / LANES; b < CHUNK / 4; b += AT_ONCE) {
                float4 q[4], w[4], a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) { q[i] = q_of(4 * b + i, d); w[i] = w_of(4 * b + i, d); a[i] = a_of(4 * b + i, d); }
                float part[16];
#pragma unroll
                for (int i = 0; i < 4; ++i) part[i] = dot4(q[i], w[i], 0.f);
                w[0] = mul4(w[0], a[1]);
                part[4] = dot4(q[1], w[0], 0.f);
                w[1] = mul4(w[1], a[2]);
                part[5] = dot4(q[2], w[1], 0.f);
                w[2] = mul4(w[2], a[3]);
                part[6] = dot4(q[3], w[2], 0.f);
                w[0] = mul4(w[0], a[2]);
                part[7] = dot4(q[2], w[0], 0.f);
                w[1] = mul4(w[1], a[3]);
                part[8] = dot4(q[3], w[1], 0.f);
                w[0] = mul4(w[0], a[3]);
                part[9] = dot4(q[3], w[0], 0.f);
#pragma unroll
                for (int i = 10; i < 16; ++i) part[i] = 0.f;
                float4 run = a[0];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    st4(qs + (4 * b + i) * LD + d, mul4(q[i], run));
                    st4(ws + (4 * b + i) * LD + d, w[i]);
                    if (i < 3) run = mul4(run, a[i + 1]);
                }
                st4(quad + b * DIM + d, run);
                // the ten sums over the row's lanes at once: every exchange halves what a lane still holds
                int held = 16;
#pragma unroll
                for (int off = LANES / 2; off > 0; off >>= 1) {
                    if (held > 1) {
                        held >>= 1;
                        const bool high = lane & off;
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            if (k < held) {
                                float send = high ? part[k] : part[k + held], keep = high ? part[k + held] : part[k];
                                part[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                            }
                        }
                    } else {
                        part[0] += __shfl_xor_sync(0xffffffffu, part[0], off);
                    }
                }
                const int sum = LANES == 32 ? lane >> 1 : lane & 15;
                if (sum < 10 && (LANES == 16 || !(lane & 1))) {
                    const int i = (int)(0x3323213210ull >> (4 * sum)) & 15, j = (int)(0x0102103210ull >> (4 * sum)) & 15;
                    A[at(4 * b + i, 4 * b + j)] = part[0];
                }
            }
        }
        __syncthreads();
        const int g = lane >> 2, t2 = (lane & 3) * 2;
        auto plain = [](float2 v, int) { return v; };
        auto plain_a = [](float2 v, int, int) { return v; };
        {
            // inside the groups of 16: the fours next to each other (a warp), and the second eight with the first (a warp)
            const int group = warp >> 1, r0 = group * GROUP;
            const float* qg = qs + r0 * LD;
            const float* wg = ws + r0 * LD;
            if (warp & 1) {
                const float *t1 = quad + (group * 4 + 1) * DIM, *t2p = quad + (group * 4 + 2) * DIM;
                float acc[1][4] = {};
                tile_product<DIM, 1>(acc, qg, LD, wg, LD,
                                  [&](float2 v, int half, int k) {
                                      const float2 f = ld2(t2p + k);
                                      return half && g >= 4 ? make_float2(v.x * f.x, v.y * f.y) : v;
                                  },
                                  [&](float2 v, int k) {
                                      const float2 f = ld2(t1 + k);
                                      return g < 4 ? make_float2(v.x * f.x, v.y * f.y) : v;
                                  });
                A[at(r0 + 8 + g, r0 + t2)] = acc[0][2];
                A[at(r0 + 8 + g, r0 + t2 + 1)] = acc[0][3];
            } else {
                float acc[2][4] = {};
                tile_product<DIM, 2>(acc, qg, LD, wg, LD, plain_a, plain);
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    if (g >= 4 && t2 < 4) {
                        A[at(r0 + 8 * half + g, r0 + 8 * half + t2)] = acc[half][2 * half];
                        A[at(r0 + 8 * half + g, r0 + 8 * half + t2 + 1)] = acc[half][2 * half + 1];
                    }
            }
        }
        __syncthreads();
        // running products over the groups' fours: half of the threads take q, half w
        for (int i = tid; i < 2 * 4 * LANES; i += THREADS) {
            const int side = i / (4 * LANES), group = (i / LANES) & 3, d = (i % LANES) * 4;
            const float* t = quad + group * 4 * DIM + d;
            float* x = (side ? ws : qs) + group * GROUP * LD + d;
            float4 run = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                run = mul4(run, ld4(t + (side ? 3 - b : b) * DIM));
                float* r = x + (side ? 2 - b : b + 1) * 4 * LD;
#pragma unroll
                for (int k = 0; k < 4; ++k) st4(r + k * LD, mul4(ld4(r + k * LD), run));
            }
            if (!side) st4(total + group * DIM + d, mul4(run, ld4(t + 3 * DIM)));
        }
        __syncthreads();
        // between groups: a warp takes one of the six 16 x 16 blocks below the diagonal; the two left multiply the groups' decays up
        if (warp < 6) {
            const int bi = warp < 1 ? 1 : warp < 3 ? 2 : 3, bj = warp - bi * (bi - 1) / 2;  // (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
            const float *m1 = total + DIM, *m2 = total + 2 * DIM;
            const int mids = bi - bj - 1;  // 0, 1 or 2 whole groups between
            const float* first = bj == 0 ? m1 : m2;
            auto of_a = [&](float2 v, int, int k) {
                if (mids > 0) { const float2 f = ld2(first + k); v = make_float2(v.x * f.x, v.y * f.y); }
                if (mids > 1) { const float2 f = ld2(m2 + k); v = make_float2(v.x * f.x, v.y * f.y); }
                return v;
            };
            float acc[2][4] = {};
            tile_product<DIM, 2>(acc, qs + bi * GROUP * LD, LD, ws + bj * GROUP * LD, LD, of_a, plain);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = bi * GROUP + g, j = bj * GROUP + 8 * half + t2;
                A[at(i, j)] = acc[half][0];
                A[at(i, j + 1)] = acc[half][1];
                A[at(i + 8, j)] = acc[half][2];
                A[at(i + 8, j + 1)] = acc[half][3];
            }
        } else {
            for (int d = tid - 6 * 32; d < DIM; d += 64) {
                float run = 1.f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    ahead[k * DIM + d] = run;
                    run *= total[k * DIM + d];
                }
            }
        }
        __syncthreads();
    }
};

// What the delta rule's chain reads of a chunk: W [64][DIM + 8], R [64][DIM + 4] and the chunk's decays [DIM].
template <int DIM> constexpr int wr_floats() { return CHUNK * (2 * DIM + 12) + DIM; }

// What the scores need of shared memory, in floats: q, w, the fours', the groups' and the earlier groups' decays, and A.
template <int DIM, bool TRANS> constexpr int scores_floats() { return 2 * CHUNK * along<DIM>() + 24 * DIM + CHUNK * Scores<DIM, TRANS>::A_LD; }

// How eight warps share a result of ROWS x COLS: 32 rows and 8 NT columns a warp.  The columns of a warp's NT tiles alternate, so that a
// lane's values of a row of the right factor, and of a row of the result, are neighbours: 2 NT of them from column `col` on.
template <int ROWS, int COLS>
struct Shares {
    static constexpr int WM = ROWS / 32, WN = THREADS / 32 / WM, WIDE = COLS < 32 * WN ? COLS : 32 * WN, NT = WIDE / (8 * WN);
    static_assert(WM * WN == THREADS / 32 && (NT == 2 || NT == 4) && COLS % WIDE == 0, "");
};
template <int NT> __device__ __forceinline__ void load_right(float (&v)[NT], const float* p) {
    if (NT == 4) { const float4 x = ld4(p); v[0] = x.x; v[1] = x.y; v[2 % NT] = x.z; v[3 % NT] = x.w; }
    else { const float2 x = ld2(p); v[0] = x.x; v[1] = x.y; }
}
// acc[2 tiles of 16 rows][NT tiles of 8 columns] += 16 of k: left(h) fills the lane's values of both row tiles for k h + 2t, h + 2t + 1 (h = 0 or 8);
// right: rows of k, `ld` apart, at the lane's own k and column.
template <int NT, typename L>
__device__ __forceinline__ void product16(float (&acc)[2][NT][4], L left, const float* right, int ld, bool both = true) {
    Two a[2][2][4], b[NT][2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float av[2][4], b0[NT], b1[NT];
        left(av, 8 * h);
        load_right<NT>(b0, right + 8 * h * ld);
        load_right<NT>(b1, right + (8 * h + 1) * ld);
#pragma unroll
        for (int n = 0; n < NT; ++n) two(b0[n], b1[n], b[n][h][0], b[n][h][1]);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            two(av[m][0], av[m][1], a[m][h][0], a[m][h][1]);
            two(av[m][2], av[m][3], a[m][h][2], a[m][h][3]);
        }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (m == 0 && !both) continue;  // (only the second tile of rows)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float c[4];
            mma6(c, a[m], b[n]);
            add_to(acc[m][n], c);
        }
    }
}

// grid: (chunks, heads, blocks of CB columns).  add: [chunks, heads, dim, vdim], fade: [chunks, heads, dim], ones: [chunks, heads, dim]
// (the normaliser's column, if cols > vdim).  q, w: head / heads_per_unit in head's place.
template <int DIM, int CB>
__global__ void __launch_bounds__(THREADS, 2)
chunk_state_kernel(const float* __restrict__ a, int a_ld, const float* __restrict__ w, int w_ld, const float* __restrict__ gates,
                   int gate_stride, const float* __restrict__ v, int v_ld, const int* __restrict__ cu_q, int num_seqs,
                   int heads, int heads_per_unit, int dim, int vdim, int cols, float* __restrict__ add,
                   float* __restrict__ fade, float* __restrict__ ones) {
    extern __shared__ __align__(16) float sm[];
    float* ws = sm;                 // [64][DIM]
    float* us = ws + CHUNK * DIM;   // [64][CB]
    float* rest = us + CHUNK * CB;  // [THREADS]
    float* bs = rest + THREADS;     // [64]
    ie_pdl_wait();
    ie_pdl_trigger();  // (chunk_out reads what was there before this kernel without waiting for it: see there)
    int seq, chunk;
    const int head = blockIdx.y, c0 = blockIdx.z * CB, tid = threadIdx.x;
    if (!find_chunk(cu_q, num_seqs, blockIdx.x, seq, chunk)) return;
    const int n0 = cu_q[seq] + chunk * CHUNK, cnt = min(CHUNK, cu_q[seq + 1] - n0);
    const size_t place = (size_t)blockIdx.x * heads + head;
    fetch_rows<CHUNK, CB, CB>(us, v + (size_t)n0 * v_ld + head * vdim + c0, v_ld, cnt, vdim - c0);
    cp_commit();
    const float* g = gates != nullptr ? gates + (size_t)n0 * gate_stride + head * 3 : nullptr;
    if (tid < CHUNK) bs[tid] = g != nullptr && tid < cnt ? g[tid * gate_stride + 1] : 0.f;
    // w_j times the decays after j: a column per thread, DIM / 256 of the chunk's tokens
    constexpr int PARTS = THREADS / DIM, EACH = CHUNK / PARTS;
    const int d = tid % DIM, part = tid / DIM;
    const float* wp = w + (size_t)n0 * w_ld + (head / heads_per_unit) * dim + d;
    const float* ap = a + (size_t)n0 * a_ld + head * dim + d;  // (not read with gates)
    float run = 1.f;
    {
        float wv[EACH], av[EACH];  // (all on their way at once: 513 tokens of 8 heads of 128 x 128 18 us by sixteens, 12.5 so)
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
            int j = (part + 1) * EACH - 1 - i;
            bool there = j < cnt && d < dim;
            wv[i] = there ? wp[(size_t)j * w_ld] : 0.f;
            av[i] = there ? (g != nullptr ? g[j * gate_stride] : ap[(size_t)j * a_ld]) : 1.f;
        }
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
            ws[((part + 1) * EACH - 1 - i) * DIM + d] = wv[i] * run;
            run *= av[i];
        }
    }
    rest[part * DIM + d] = run;
    __syncthreads();
    float after = 1.f, whole = 1.f;
#pragma unroll
    for (int p = PARTS - 1; p >= 0; --p) {
        if (p == part) after = whole;
        whole *= rest[p * DIM + d];
    }
    if (part + 1 < PARTS)
        for (int j = part * EACH; j < (part + 1) * EACH; ++j) ws[j * DIM + d] *= after;
    if (part == 0 && c0 == 0 && d < dim) fade[place * dim + d] = whole;
    cp_wait<0>();
    __syncthreads();
    if (g != nullptr) {  // u = gate * v
        for (int i = tid; i < CHUNK * CB; i += THREADS) us[i] *= bs[i / CB];
        __syncthreads();
    }
    if (cols > vdim && c0 == 0 && part == 0 && d < dim) {
        float s = 0.f;
        for (int j = 0; j < CHUNK; ++j) s = fmaf(ws[j * DIM + d], bs[j], s);
        ones[place * dim + d] = s;
    }
    // [DIM x 64] [64 x CB]: a thread holds ROWS consecutive channels of four columns, two channels to an instruction (the results are
    // those of single multiply-adds.  Products put together on the tensor cores, below, would take the same 36 us of 2,048 tokens and 16 heads
    // of 128 x 128, but the decays let the terms grow towards a chain's end, where they are further off: 1.1e-7 against 0.8e-7)
    constexpr int LC = CB / 4, ROWS = DIM * LC / THREADS;
    const int lc = tid % LC, r0 = (tid / LC) * ROWS;
    unsigned long long acc[ROWS / 2][4];
#pragma unroll
    for (int r = 0; r < ROWS / 2; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0ull;
#pragma unroll 2
    for (int j = 0; j < CHUNK; ++j) {
        const float4 u = ld4(us + j * CB + lc * 4);
        const unsigned long long uv[4] = {packed(u.x, u.x), packed(u.y, u.y), packed(u.z, u.z), packed(u.w, u.w)};
#pragma unroll
        for (int r = 0; r < ROWS; r += 4) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(ws + j * DIM + r0 + r);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r / 2][k]) : "l"(x.x), "l"(uv[k]));
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r / 2 + 1][k]) : "l"(x.y), "l"(uv[k]));
            }
        }
    }
    const int c = c0 + lc * 4;
    if (c >= vdim) return;
#pragma unroll
    for (int r = 0; r < ROWS; r += 2) {
        float2 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[k].x), "=f"(v[k].y) : "l"(acc[r / 2][k]));
        if (r0 + r < dim) st4(add + (place * dim + r0 + r) * vdim + c, make_float4(v[0].x, v[1].x, v[2].x, v[3].x));
        if (r0 + r + 1 < dim) st4(add + (place * dim + r0 + r + 1) * vdim + c, make_float4(v[0].y, v[1].y, v[2].y, v[3].y));
    }
}

// grid: (blocks of eight warps, a warp takes eight channels of sixteen columns, and one block for the normaliser's column; heads;
// requests).  So the scratch is read in pieces of 64 bytes and the slot, which holds columns, in pieces of 32.  A chain of `chunks` loads,
// multiplies and stores per entry: the next eight chunks' sums are on their way (four: 23 us for 32 chunks of 16 heads).
__global__ void __launch_bounds__(THREADS)
chunk_scan_kernel(float* __restrict__ add, const float* __restrict__ fade, float* __restrict__ ones, float* __restrict__ state,
                  long long state_stride, const int* __restrict__ slots, const int* __restrict__ cu_q, int heads, int dim,
                  int vdim, int cols, int num_slots) {
    ie_pdl_trigger();
    ie_pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z, len = cu_q[seq + 1] - cu_q[seq], slot = slots[seq];
    if (len <= 0 || slot < 0 || slot >= num_slots) return;
    int first = 0;  // the request's first chunk among the step's
    for (int s = 0; s < seq; ++s) first += (cu_q[s + 1] - cu_q[s] + CHUNK - 1) / CHUNK;
    const int chunks = (len + CHUNK - 1) / CHUNK;
    float* S = state + (size_t)slot * state_stride + (size_t)head * cols * dim;
    const size_t place = (size_t)first * heads + head;
    constexpr int AHEAD = 8;
    if (cols > vdim && blockIdx.x + 1 == gridDim.x) {
        for (int d = threadIdx.x; d < dim; d += THREADS) {
            float s = S[(size_t)vdim * dim + d];
            for (int c = 0; c < chunks; ++c) {
                size_t at = (place + (size_t)c * heads) * dim + d;
                float x = ones[at];
                ones[at] = s;
                s = fmaf(fade[at], s, x);
            }
            S[(size_t)vdim * dim + d] = s;
        }
        return;
    }
    const int across = (vdim + 15) / 16, tile = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int d = (tile / across) * 8 + (lane >> 2), col = (tile % across) * 16 + (lane & 3) * 4;
    if (d >= dim || col >= vdim) return;
    float* p = add + (place * dim + d) * vdim + col;
    const float* f = fade + place * dim + d;
    const size_t p_step = (size_t)heads * dim * vdim, f_step = (size_t)heads * dim;
    float* at = S + (size_t)col * dim + d;
    float4 s = make_float4(at[0], at[dim], at[2 * dim], at[3 * dim]);
    float4 x[AHEAD];
    float y[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
        if (i < chunks) { x[i] = ld4(p + i * p_step); y[i] = f[i * f_step]; }
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            int c = c0 + i;
            if (c < chunks) {
                float4 xi = x[i];
                float yi = y[i];
                if (c + AHEAD < chunks) { x[i] = ld4(p + (c + AHEAD) * p_step); y[i] = f[(c + AHEAD) * f_step]; }
                st4(p + c * p_step, s);
                s = make_float4(fmaf(yi, s.x, xi.x), fmaf(yi, s.y, xi.y), fmaf(yi, s.z, xi.z), fmaf(yi, s.w, xi.w));
            }
        }
    }
    at[0] = s.x;
    at[dim] = s.y;
    at[2 * dim] = s.z;
    at[3 * dim] = s.w;
}

// grid: (chunks, heads, blocks of CB columns).  before: the state before each chunk, [chunks, heads, dim, vdim]; ones: its
// normaliser's column.  u: element (n, head, c) at [n * u_ld + head * vdim + c], or with `own` [chunks, heads, 64, vdim].
// out: [N, heads, cols], times q_scale.  100 KB of shared memory, two blocks per SM: once the scores stand, the state and then u come in
// pieces of 32 rows, two at a time, where w was.
// Parts of a product that are subtracted from one another make no number of an infinite one: scores and outputs that come out without a finite value are
// formed again, one multiply-add after the other.
template <int DIM, int CB>
__global__ void __launch_bounds__(THREADS, 2)
chunk_out_kernel(const float* __restrict__ q, int q_ld, const float* __restrict__ a, int a_ld, const float* __restrict__ w,
                 int w_ld, const float* __restrict__ gates, int gate_stride, const float* __restrict__ u, int u_ld, int own,
                 const float* __restrict__ before, const float* __restrict__ ones, const int* __restrict__ slots,
                 const int* __restrict__ cu_q, int num_seqs, float* __restrict__ out, int heads, int heads_per_unit, int dim,
                 int vdim, int cols, float q_scale, int num_slots) {
    using Sc = Scores<DIM, false>;
    constexpr int LD = Sc::LD, LB = CB + 4, PIECE = 32;
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                         // [64][DIM + 8]
    float* A = qs + CHUNK * LD;             // [64][72]
    float* total = A + CHUNK * Sc::A_LD;    // [4][DIM]
    float* ahead = total + 4 * DIM;         // [4][DIM]
    float* ws = ahead + 4 * DIM;            // [64][DIM + 8], then the pieces: two of [32][CB + 4]
    float* quad = ws + CHUNK * LD;          // [16][DIM]
    ie_pdl_trigger();
    // The scores need nothing of the two kernels before, chunk_state and chunk_scan or the delta rule's two, and so do not wait for them: the first
    // of those lets the second start, and that one this, only once all that ran before is done.  (Scores formed meanwhile: 513 tokens of 8 heads 22 us after them, 18 so; 2,048 of the delta rule's 16, whose chain leaves 20 SMs idle, 70 and 61.)
    int seq, chunk;
    const int head = blockIdx.y, c0 = blockIdx.z * CB, tid = threadIdx.x, unit = head / heads_per_unit;
    const bool there = find_chunk(cu_q, num_seqs, blockIdx.x, seq, chunk);
    const int slot = there ? slots[seq] : -1;
    if (slot < 0 || slot >= num_slots) {
        ie_pdl_wait();  // (what runs next waits for this kernel alone: it is not done before those are)
        return;
    }
    const int n0 = cu_q[seq] + chunk * CHUNK, cnt = min(CHUNK, cu_q[seq + 1] - n0);
    const size_t place = (size_t)blockIdx.x * heads + head;
    const float* g = gates != nullptr ? gates + (size_t)n0 * gate_stride + head * 3 : nullptr;
    const float *qp = q + (size_t)n0 * q_ld + unit * dim, *wp = w + (size_t)n0 * w_ld + unit * dim, *ap = a + (size_t)n0 * a_ld + head * dim;
    const float4 zeros = make_float4(0.f, 0.f, 0.f, 0.f), ones4 = make_float4(1.f, 1.f, 1.f, 1.f);
    Sc::run(qs, ws, quad, total, ahead, A,
            [&](int row, int d) { return row < cnt && d < dim ? ld4(qp + (size_t)row * q_ld + d) : zeros; },
            [&](int row, int d) { return row < cnt && d < dim ? ld4(wp + (size_t)row * w_ld + d) : zeros; },
            [&](int row, int d) {
                if (row >= cnt) return ones4;
                if (g != nullptr) { const float f = g[row * gate_stride]; return make_float4(f, f, f, f); }
                return d < dim ? ld4(ap + (size_t)row * a_ld + d) : ones4;
            });
    // the state, then u, in pieces of 32 rows
    constexpr int STATE_PIECES = DIM / PIECE, PIECES = STATE_PIECES + CHUNK / PIECE;
    auto fetch = [&](int p) {
        float* to = ws + (p & 1) * PIECE * LB;
        if (p < STATE_PIECES) {
            fetch_rows<PIECE, CB, LB>(to, before + (place * dim + p * PIECE) * vdim + c0, vdim, dim - p * PIECE, vdim - c0);
        } else {
            const int j0 = (p - STATE_PIECES) * PIECE;
            if (own) fetch_rows<PIECE, CB, LB>(to, u + (place * CHUNK + j0) * vdim + c0, vdim, cnt - j0, vdim - c0);
            else fetch_rows<PIECE, CB, LB>(to, u + (size_t)(n0 + j0) * u_ld + head * vdim + c0, u_ld, cnt - j0, vdim - c0);
        }
        cp_commit();
    };
    ie_pdl_wait();
    fetch(0);
    fetch(1);
    if (g != nullptr) {  // u = gate * v, on the scores' side
        for (int i = tid; i < CHUNK * CHUNK; i += THREADS) {
            const int row = i / CHUNK, col = i % CHUNK;
            if (col <= row) A[Sc::at(row, col)] *= col < cnt ? g[col * gate_stride + 1] : 0.f;
        }
    }
    using Sh = Shares<CHUNK, CB>;
    static_assert(Sh::WIDE == CB, "");
    constexpr int NT = Sh::NT;
    const int warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t2 = (lane & 3) * 2;
    const int half = warp % Sh::WM, r0 = half * 32, nc = (warp / Sh::WM) * 8 * NT;
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;
#pragma unroll 1
    for (int p = 0; p < PIECES; ++p) {
        if (p + 1 < PIECES) cp_wait<1>();
        else cp_wait<0>();
        __syncthreads();
        const float* piece = ws + (p & 1) * PIECE * LB;
        if (p < STATE_PIECES) {
#pragma unroll
            for (int k = 0; k < PIECE; k += 16)
                product16<NT>(acc, [&](float (&av)[2][4], int h) {
                    const int d = p * PIECE + k + h + t2;
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        const float2 f = ld2(ahead + (r0 / 16 + m) * DIM + d);
                        const float2 x = ld2(qs + (r0 + 16 * m + g8) * LD + d), y = ld2(qs + (r0 + 16 * m + 8 + g8) * LD + d);
                        av[m][0] = x.x * f.x; av[m][1] = y.x * f.x; av[m][2] = x.y * f.y; av[m][3] = y.y * f.y;
                    }
                }, piece + (k + t2) * LB + nc + NT * g8, LB);
        } else {
            const int jp = p - STATE_PIECES, j0 = jp * PIECE;
            if (half >= jp) {  // tokens before the tile's own 16
                const bool both = half > jp;
#pragma unroll 1
                for (int k = 0; k < (both ? PIECE : 16); k += 16)
                    product16<NT>(acc, [&](float (&av)[2][4], int h) {
                        const int j = j0 + k + h + t2;
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            const float2 x = ld2(A + Sc::at(r0 + 16 * m + g8, j)), y = ld2(A + Sc::at(r0 + 16 * m + 8 + g8, j));
                            av[m][0] = x.x; av[m][1] = y.x; av[m][2] = x.y; av[m][3] = y.y;
                        }
                    }, piece + (k + t2) * LB + nc + NT * g8, LB, both);
            }
            if (half == jp) {  // and its own, the triangle: no token reads a later one's value, whatever it is
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const float *a0 = A + Sc::at(r0 + 16 * m + g8, r0 + 16 * m), *a1 = a0 + 8 * Sc::A_LD, *up = piece + 16 * m * LB + nc + NT * t2;
#pragma unroll 1
                    for (int j4 = 0; j4 < 16; j4 += 4) {
                      const float4 xs = ld4(a0 + j4), ys = ld4(a1 + j4);
                      const float xv[4] = {xs.x, xs.y, xs.z, xs.w}, yv[4] = {ys.x, ys.y, ys.z, ys.w};
#pragma unroll
                      for (int jj = 0; jj < 4; ++jj) {
                        const int j = j4 + jj;
                        const float x = xv[jj], y = yv[jj];
                        float uv[2 * NT];
#pragma unroll
                        for (int k = 0; k < 2 * NT; k += 4) {
                            const float4 v4 = ld4(up + j * LB + k);
                            uv[k] = v4.x; uv[k + 1] = v4.y; uv[k + 2] = v4.z; uv[k + 3] = v4.w;
                        }
                        if (j <= g8)
#pragma unroll
                            for (int n = 0; n < NT; ++n) {
                                acc[m][n][0] = fmaf(x, uv[n], acc[m][n][0]);
                                acc[m][n][1] = fmaf(x, uv[NT + n], acc[m][n][1]);
                            }
                        if (j <= g8 + 8)
#pragma unroll
                            for (int n = 0; n < NT; ++n) {
                                acc[m][n][2] = fmaf(y, uv[n], acc[m][n][2]);
                                acc[m][n][3] = fmaf(y, uv[NT + n], acc[m][n][3]);
                            }
                      }
                    }
                }
            }
        }
        __syncthreads();
        if (p + 2 < PIECES) fetch(p + 2);
    }
    const int c = c0 + nc + NT * t2;  // 2 NT columns from here on
    auto no_number = [](float x) { return !(fabsf(x) <= FLT_MAX); };
    bool odd = false;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = r0 + 16 * m + 8 * r + g8;
            if (row >= cnt) continue;
            float* to = out + ((size_t)(n0 + row) * heads + head) * cols + c;
            float o[2 * NT];
#pragma unroll
            for (int n = 0; n < NT; ++n) { o[n] = acc[m][n][2 * r] * q_scale; o[NT + n] = acc[m][n][2 * r + 1] * q_scale; }
#pragma unroll
            for (int k = 0; k < 2 * NT; k += 4) {
                if (c + k >= vdim) break;
                odd |= no_number(o[k]) || no_number(o[k + 1]) || no_number(o[k + 2]) || no_number(o[k + 3]);
                if (cols == vdim) st4(to + k, make_float4(o[k], o[k + 1], o[k + 2], o[k + 3]));
                else { to[k] = o[k]; to[k + 1] = o[k + 1]; to[k + 2] = o[k + 2]; to[k + 3] = o[k + 3]; }  // (rows of an odd length)
            }
        }
    if (__syncthreads_or(odd)) {
        for (int i = tid; i < CHUNK * CHUNK; i += THREADS) {
            const int row = i / CHUNK, j = i % CHUNK;
            if (j > row || row >= cnt || !no_number(A[Sc::at(row, j)])) continue;
            float s = 0.f;
            for (int d = 0; d < dim; ++d) {
                float x = qp[(size_t)row * q_ld + d];
                for (int t = j + 1; t <= row; ++t) x *= g != nullptr ? g[t * gate_stride] : ap[(size_t)t * a_ld + d];
                s = fmaf(x, wp[(size_t)j * w_ld + d], s);
            }
            A[Sc::at(row, j)] = g != nullptr ? s * g[j * gate_stride + 1] : s;
        }
        __syncthreads();
        for (int i = tid; i < cnt * CB; i += THREADS) {
            const int row = i / CB, col = c0 + i % CB;
            float* to = out + ((size_t)(n0 + row) * heads + head) * cols + col;
            if (col >= vdim || !no_number(*to)) continue;
            float s = 0.f;
            for (int d = 0; d < dim; ++d) s = fmaf(qs[row * LD + d] * ahead[row / GROUP * DIM + d], before[(place * dim + d) * vdim + col], s);
            for (int j = 0; j <= row; ++j)
                s = fmaf(A[Sc::at(row, j)], own ? u[(place * CHUNK + j) * vdim + col] : u[(size_t)(n0 + j) * u_ld + head * vdim + col], s);
            *to = s * q_scale;
        }
    }
    if (cols > vdim && c0 == 0) {  // the normaliser's column, whose values are the gates
        for (int i = warp; i < cnt; i += THREADS / 32) {
            float s = 0.f;
            for (int d = lane; d < dim; d += 32) s = fmaf(qs[i * LD + d] * ahead[i / GROUP * DIM + d], ones[place * dim + d], s);
            for (int j = lane; j <= i; j += 32) s += A[Sc::at(i, j)];
            s = warp_sum(s);
            if (lane == 0) out[((size_t)(n0 + i) * heads + head) * cols + vdim] = s * q_scale;
        }
    }
}

// Both right-hand sides by forward substitution, a column per thread: x[i] -= L(i, j) x[j].  Lt: [j][i] with 72 between.
__device__ __forceinline__ void substitute(float (&x)[CHUNK], const float* Lt) {
#pragma unroll
    for (int j = 0; j < CHUNK - 1; ++j) {
#pragma unroll
        for (int p = (j + 1) / 4; p < CHUNK / 4; ++p) {
            float4 l = ld4(Lt + j * (CHUNK + 8) + 4 * p);
            const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (4 * p + i > j) x[4 * p + i] = fmaf(-lv[i], x[j], x[4 * p + i]);
        }
    }
}

// grid: (chunks, heads).  U: [chunks, heads, 64, vdim]; WR: per chunk and head what the chain reads (`wr_floats`): W, the keys times the
// decays after them, the chunk's decays.
// The substitution goes 16 tokens at a time: the tokens before them by products on the tensor cores, then the inverse of their own
// triangle times what is left, a warp 32 columns of W or U.  (A column a thread through all 64 tokens is 2,600 instructions that every warp
// executes once: a third of the time went on fetching them.)  In such products a value that is no number would reach the tokens before it; a chunk that
// has one goes token by token.
template <int DIM>
__global__ void __launch_bounds__(THREADS, 2)
delta_solve_kernel(const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ beta,
                   const float* __restrict__ decay, const int* __restrict__ cu_q, int num_seqs, int heads, int kv_heads,
                   int dim, int vdim, float* __restrict__ U, float* __restrict__ WR) {
    using Sc = Scores<DIM, true>;
    constexpr int LD = Sc::LD, LL = Sc::A_LD, LI = 24, LR = DIM + 4;
    constexpr int VC = 128, LV = VC + 8;      // columns of U, and between its rows
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                           // [64][DIM + 8], then W
    float* Lt = qs + CHUNK * LD;              // [j][i]
    float* total = Lt + CHUNK * LL;           // [4][DIM]
    float* ahead = total + 4 * DIM;           // [4][DIM]
    float* bs = ahead + 4 * DIM;              // [64]
    float* inv = bs + CHUNK;                  // [4][16][24]: the groups' inverses, [j][i]
    float* ws = inv + 4 * GROUP * LI;         // [64][DIM + 8], then U [64][136]
    float* quad = ws + CHUNK * LD;            // [16][DIM]
    ie_pdl_wait();
    ie_pdl_trigger();  // (as in chunk_state)
    int seq, chunk;
    const int head = blockIdx.y, tid = threadIdx.x, kvh = head / (heads / kv_heads);
    if (!find_chunk(cu_q, num_seqs, blockIdx.x, seq, chunk)) return;
    const int n0 = cu_q[seq] + chunk * CHUNK, cnt = min(CHUNK, cu_q[seq + 1] - n0);
    const size_t place = (size_t)blockIdx.x * heads + head;
    const float* kp = k + ((size_t)n0 * kv_heads + kvh) * dim;
    const float* ap = decay + ((size_t)n0 * heads + head) * dim;
    const float* vp = v + ((size_t)n0 * heads + head) * vdim;
    float* W = WR + place * wr_floats<DIM>();
    float* R = W + CHUNK * LD;
    U += place * CHUNK * vdim;
    if (tid < CHUNK) bs[tid] = tid < cnt ? beta[(size_t)(n0 + tid) * heads + head] : 0.f;
    const float4 zeros = make_float4(0.f, 0.f, 0.f, 0.f), ones4 = make_float4(1.f, 1.f, 1.f, 1.f);
    auto key = [&](int row, int d) { return row < cnt && d < dim ? ld4(kp + (size_t)row * kv_heads * dim + d) : zeros; };
    auto fade = [&](int row, int d) { return row < cnt && d < dim ? ld4(ap + (size_t)row * heads * dim + d) : ones4; };
    Sc::run(qs, ws, quad, total, ahead, Lt, key, key, fade);
    // the keys that the state's update takes, and the chunk's decays
    for (int i = tid; i < CHUNK * DIM / 4; i += THREADS) {
        const int row = i / (DIM / 4), d = i % (DIM / 4) * 4, g = row / GROUP;
        float4 x = ld4(ws + row * LD + d);
        for (int m = g + 1; m < CHUNK / GROUP; ++m) x = mul4(x, ld4(total + m * DIM + d));
        st4(R + row * LR + d, x);
    }
    if (tid < DIM) R[CHUNK * LR + tid] = ahead[3 * DIM + tid] * total[3 * DIM + tid];
    __syncthreads();
    // rows times beta, on both sides
    bool odd = false;  // a value that is no number, or beyond all
    auto see = [&](float4 x) { odd |= !(fabsf(x.x) <= FLT_MAX && fabsf(x.y) <= FLT_MAX && fabsf(x.z) <= FLT_MAX && fabsf(x.w) <= FLT_MAX); };
    for (int i = tid; i < CHUNK * DIM / 4; i += THREADS) {
        const int row = i / (DIM / 4), d = i % (DIM / 4) * 4;
        const float f = bs[row];
        const float4 x = mul4(mul4(ld4(qs + row * LD + d), ld4(ahead + row / GROUP * DIM + d)), make_float4(f, f, f, f));
        see(x);
        st4(qs + row * LD + d, x);
    }
    for (int i = tid; i < CHUNK * VC / 4; i += THREADS) {
        const int row = i / (VC / 4), c = i % (VC / 4) * 4;
        const float f = bs[row];
        const float4 x = row < cnt && c < vdim ? mul4(ld4(vp + (size_t)row * heads * vdim + c), make_float4(f, f, f, f)) : zeros;
        see(x);
        st4(ws + row * LV + c, x);
    }
    for (int i = tid; i < CHUNK * CHUNK; i += THREADS) {
        const int j = i / CHUNK, row = i % CHUNK;
        if (row > j) Lt[j * LL + row] *= bs[row];
    }
    odd = __syncthreads_or(odd);
    if (!odd && tid < CHUNK) {  // a column of a group's inverse per thread
        const int g = tid / GROUP, c = tid % GROUP;
        float x[GROUP];
#pragma unroll
        for (int i = 0; i < GROUP; ++i) x[i] = i == c ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < GROUP - 1; ++j)
#pragma unroll
            for (int i = j + 1; i < GROUP; ++i) x[i] = fmaf(-Lt[(g * GROUP + j) * LL + g * GROUP + i], x[j], x[i]);
#pragma unroll
        for (int i = 0; i < GROUP; ++i) inv[(g * GROUP + c) * LI + i] = i < c ? 0.f : x[i];
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t = lane & 3;
    constexpr int W_WARPS = DIM / 32;
    if (!odd && warp < W_WARPS + VC / 32) {
        const bool is_w = warp < W_WARPS;
        const int ld = is_w ? LD : LV, n0c = (is_w ? warp : warp - W_WARPS) * 32, col = n0c + 8 * t;  // the lane's eight columns of a result
        float* X = is_w ? qs : ws;
        // 16 of k: rows `left` of [j][i] (a row of j `l_ld` apart), rows `right` of X
        auto product = [&](float (&c)[4][4], const float* left, int l_ld, const float* right) {
            Two a[2][4], b[4][2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float *l0 = left + (8 * h + t) * l_ld + g8, *l1 = l0 + 4 * l_ld, *r0 = right + (8 * h + t) * ld + n0c + 4 * g8;
                two(l0[0], l0[8], a[h][0], a[h][1]);
                two(l1[0], l1[8], a[h][2], a[h][3]);
                const float4 x = ld4(r0), y = ld4(r0 + 4 * ld);
                two(x.x, y.x, b[0][h][0], b[0][h][1]);
                two(x.y, y.y, b[1][h][0], b[1][h][1]);
                two(x.z, y.z, b[2][h][0], b[2][h][1]);
                two(x.w, y.w, b[3][h][0], b[3][h][1]);
            }
#pragma unroll
            for (int n = 0; n < 4; ++n) mma6(c[n], a, b[n]);
        };
        auto put = [&](float* p, const float (&c)[4][4], int half) {
            st4(p, make_float4(c[0][2 * half], c[1][2 * half], c[2][2 * half], c[3][2 * half]));
            st4(p + 4, make_float4(c[0][2 * half + 1], c[1][2 * half + 1], c[2][2 * half + 1], c[3][2 * half + 1]));
        };
#pragma unroll 1
        for (int g = 0; g < CHUNK / GROUP; ++g) {
            float* own = X + (g * GROUP + g8) * ld + col;
            if (g > 0) {
                float acc[4][4] = {};
#pragma unroll 1
                for (int h = 0; h < g; ++h) {
                    float c[4][4];
                    product(c, Lt + h * GROUP * LL + g * GROUP, LL, X + h * GROUP * ld);
#pragma unroll
                    for (int n = 0; n < 4; ++n) add_to(acc[n], c[n]);
                }
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float* p = own + 8 * half * ld;
                    const float4 x = ld4(p), y = ld4(p + 4);
                    acc[0][2 * half] = x.x - acc[0][2 * half];
                    acc[1][2 * half] = x.y - acc[1][2 * half];
                    acc[2][2 * half] = x.z - acc[2][2 * half];
                    acc[3][2 * half] = x.w - acc[3][2 * half];
                    acc[0][2 * half + 1] = y.x - acc[0][2 * half + 1];
                    acc[1][2 * half + 1] = y.y - acc[1][2 * half + 1];
                    acc[2][2 * half + 1] = y.z - acc[2][2 * half + 1];
                    acc[3][2 * half + 1] = y.w - acc[3][2 * half + 1];
                    put(p, acc, half);
                }
                __syncwarp();
            }
            float c[4][4];
            product(c, inv + g * GROUP * LI, LI, X + g * GROUP * ld);
            __syncwarp();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int row = g * GROUP + 8 * half + g8;
                put(own + 8 * half * ld, c, half);
#pragma unroll
                for (int n = 0; n < 4; ++n) odd |= !(fabsf(c[n][2 * half]) <= FLT_MAX && fabsf(c[n][2 * half + 1]) <= FLT_MAX);
                if (is_w) put(W + row * LD + col, c, half);
                else {
                    if (col < vdim) st4(U + row * vdim + col, make_float4(c[0][2 * half], c[1][2 * half], c[2][2 * half], c[3][2 * half]));
                    if (col + 4 < vdim)
                        st4(U + row * vdim + col + 4, make_float4(c[0][2 * half + 1], c[1][2 * half + 1], c[2][2 * half + 1], c[3][2 * half + 1]));
                }
            }
            __syncwarp();
        }
    }
    if (!__syncthreads_or(odd)) return;
    // token by token, from the start
    Sc::run(qs, ws, quad, total, ahead, Lt, key, key, fade);
    for (int i = tid; i < CHUNK * CHUNK; i += THREADS) {
        const int j = i / CHUNK, row = i % CHUNK;
        if (row > j) Lt[j * LL + row] *= bs[row];
    }
    __syncthreads();
    const int c = tid - DIM;
    float x[CHUNK];
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) {
        if (c < 0) x[i] = qs[i * LD + tid] * ahead[i / GROUP * DIM + tid] * bs[i];
        else x[i] = i < cnt && c < vdim ? vp[(size_t)i * heads * vdim + c] * bs[i] : 0.f;
    }
    substitute(x, Lt);
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) {
        if (c < 0) W[i * LD + tid] = x[i];
        else if (c < vdim) U[i * vdim + c] = x[i];
    }
}

// grid: (blocks of 16 columns, heads, requests).  U becomes u; before: [chunks, heads, dim, vdim].
// What bounds it is a chunk's latency, two products one behind the other, thirty-two times for 2,048 tokens.  u = U - W S0: a warp takes
// 16 tokens and 8 columns and goes through all channels, so that no sums meet; the state after: a warp takes 16 channels (all 16 columns, or
// 8 of them with 64 channels) and keeps them in its registers, from where the next chunk's first product gets them through shared memory.
constexpr int CO = 16, U_LD = CHUNK + 8;
template <int DIM>
__global__ void __launch_bounds__(THREADS, 1)
delta_chain_kernel(float* __restrict__ U, const float* __restrict__ WR, float* __restrict__ before, float* __restrict__ state, long long state_stride, const int* __restrict__ slots,
                   const int* __restrict__ cu_q, int heads, int dim, int vdim, int num_slots) {
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = along<DIM>(), LR = DIM + 4, NTC = DIM / 64;
    float* buf = sm;                         // two chunks' W [64][DIM + 8], R [64][DIM + 4] and decays [DIM]
    float* Ss = buf + 2 * wr_floats<DIM>();  // [16][DIM + 8]: the state's columns
    float* Us = Ss + CO * LD;                // [16][72]: u's columns
    ie_pdl_trigger();
    ie_pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z, c0 = blockIdx.x * CO, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int len = cu_q[seq + 1] - cu_q[seq], slot = slots[seq];
    if (len <= 0 || slot < 0 || slot >= num_slots) return;
    int first = 0;
    for (int s = 0; s < seq; ++s) first += (cu_q[s + 1] - cu_q[s] + CHUNK - 1) / CHUNK;
    const int chunks = (len + CHUNK - 1) / CHUNK;
    const int g = lane >> 2, t2 = (lane & 3) * 2;
    float* S = state + (size_t)slot * state_stride + ((size_t)head * vdim + c0) * dim;
    // the lane's part of the state: channels d0 and d0 + 1, columns col and col + 1 of NTC tiles of 8
    const int d0 = (NTC == 2 ? warp : warp >> 1) * 16 + 2 * g, n1 = NTC == 2 ? 0 : (warp & 1) * 8;
    float st[NTC][2][2];  // [tile][channel][column]
    auto leave_state = [&]() {
#pragma unroll
        for (int n = 0; n < NTC; ++n)
#pragma unroll
            for (int c = 0; c < 2; ++c)
                *reinterpret_cast<float2*>(Ss + (n1 + 8 * n + t2 + c) * LD + d0) = make_float2(st[n][0][c], st[n][1][c]);
    };
#pragma unroll
    for (int n = 0; n < NTC; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int col = n1 + 8 * n + t2 + c;
                st[n][r][c] = c0 + col < vdim && d0 + r < dim ? S[(size_t)col * dim + d0 + r] : 0.f;
            }
    leave_state();
    auto fetch = [&](int c) {
        const float* from = WR + ((size_t)(first + c) * heads + head) * wr_floats<DIM>() + 4 * tid;
        float* to = buf + (c & 1) * wr_floats<DIM>() + 4 * tid;
#pragma unroll
        for (int i = 0; i < (wr_floats<DIM>() + 4 * THREADS - 1) / (4 * THREADS); ++i)
            if ((i + 1) * 4 * THREADS <= wr_floats<DIM>() || 4 * tid + i * 4 * THREADS < wr_floats<DIM>())
                cp16(to + i * 4 * THREADS, from + i * 4 * THREADS, true);
        cp_commit();
    };
    fetch(0);
    const int row = (warp >> 1) * 16 + g, ucol = (warp & 1) * 8 + t2;  // the lane's u: this row and the eighth after it, two columns
    const bool ucols = c0 + ucol < vdim;
    for (int c = 0; c < chunks; ++c) {
        const float *Wb = buf + (c & 1) * wr_floats<DIM>(), *Rb = Wb + CHUNK * LD, *Ps = Rb + CHUNK * LR;
        const size_t place = (size_t)(first + c) * heads + head;
        cp_wait<0>();
        __syncthreads();  // the chunk's W and R, the state; and nobody reads the other buffers any more
        if (c + 1 < chunks) fetch(c + 1);
        float* up = U + (place * CHUNK + row) * vdim + c0 + ucol;
        const float2 none = make_float2(0.f, 0.f), u0 = ucols ? ld2(up) : none, u1 = ucols ? ld2(up + 8 * vdim) : none;
        // the state before the chunk, for the outputs
#pragma unroll
        for (int n = 0; n < NTC; ++n)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int col = c0 + n1 + 8 * n + t2;
                if (d0 + r < dim && col < vdim)
                    *reinterpret_cast<float2*>(before + (place * dim + d0 + r) * vdim + col) = make_float2(st[n][r][0], st[n][r][1]);
            }
        {
            float acc[1][4] = {};
            tile_product<DIM, 1>(acc, Wb + (warp >> 1) * 16 * LD, LD, Ss + (warp & 1) * 8 * LD, LD,
                                 [](float2 v, int, int) { return v; }, [](float2 v, int) { return v; });
            const float2 v0 = make_float2(u0.x - acc[0][0], u0.y - acc[0][1]), v1 = make_float2(u1.x - acc[0][2], u1.y - acc[0][3]);
            Us[ucol * U_LD + row] = v0.x;
            Us[(ucol + 1) * U_LD + row] = v0.y;
            Us[ucol * U_LD + row + 8] = v1.x;
            Us[(ucol + 1) * U_LD + row + 8] = v1.y;
            if (ucols) {
                *reinterpret_cast<float2*>(up) = v0;
                *reinterpret_cast<float2*>(up + 8 * vdim) = v1;
            }
        }
        __syncthreads();
        {
            float acc[NTC][4];
#pragma unroll
            for (int n = 0; n < NTC; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
            const float* rb = Rb + d0;
#pragma unroll 2
            for (int j = 0; j < CHUNK; j += 16) {
                Two a[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 x = ld2(rb + (j + 8 * h + t2) * LR), y = ld2(rb + (j + 8 * h + t2 + 1) * LR);
                    two(x.x, x.y, a[h][0], a[h][1]);
                    two(y.x, y.y, a[h][2], a[h][3]);
                }
#pragma unroll
                for (int n = 0; n < NTC; ++n) {
                    Two b[2][2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float2 z = ld2(Us + (n1 + 8 * n + g) * U_LD + j + 8 * h + t2);
                        two(z.x, z.y, b[h][0], b[h][1]);
                    }
                    float cc[4];
                    mma6(cc, a, b);
                    add_to(acc[n], cc);
                }
            }
            const float2 f = ld2(Ps + d0);
#pragma unroll
            for (int n = 0; n < NTC; ++n)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    st[n][0][i] = fmaf(f.x, st[n][0][i], acc[n][i]);
                    st[n][1][i] = fmaf(f.y, st[n][1][i], acc[n][2 + i]);
                }
            leave_state();
        }
    }
#pragma unroll
    for (int n = 0; n < NTC; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int col = n1 + 8 * n + t2 + c;
                if (c0 + col < vdim && d0 + r < dim) S[(size_t)col * dim + d0 + r] = st[n][r][c];
            }
}

template <int DIM, int CB> constexpr size_t out_smem() {
    const int scores = scores_floats<DIM, false>(), pieces = CHUNK * along<DIM>() + CHUNK * Scores<DIM, false>::A_LD + 8 * DIM + 2 * 32 * (CB + 4);
    return (size_t)(scores > pieces ? scores : pieces) * sizeof(float);
}
template <int DIM> constexpr size_t solve_smem() {
    const int used = DIM == 128 ? CHUNK * along<DIM>() + 16 * DIM : CHUNK * 136;  // w and the fours' decays, then U
    return (size_t)(CHUNK * along<DIM>() + CHUNK * Scores<DIM, true>::A_LD + 8 * DIM + CHUNK + 4 * GROUP * 24 + used) * sizeof(float);
}
constexpr size_t state_smem(int dim, int cb) { return (size_t)(CHUNK * (dim + cb) + THREADS + CHUNK) * sizeof(float); }
template <int DIM> constexpr size_t chain_smem() {
    return (size_t)(2 * wr_floats<DIM>() + CO * (along<DIM>() + U_LD)) * sizeof(float);
}

struct Args {
    const float *q, *a, *w, *gates, *v;
    int q_ld, a_ld, w_ld, gate_stride, v_ld;
    float* state;
    long long state_stride;
    const int *slots, *cu_q;
    float* out;
    int num_seqs, heads, heads_per_unit, dim, vdim, cols;
    float q_scale;
    int num_slots, chunks;
    cudaStream_t s;
};

// Blocks of 128 columns form the chunk's scores once for all of them; with so few blocks that the device would idle, two of 64
// columns are done sooner.
bool wide_blocks(const Args& t) { return t.vdim > 64 && t.chunks * t.heads > ie_sm_count(); }

template <int DIM, int CB>
int launch_out(const Args& t, const float* u, int u_ld, int own, const float* before, const float* ones) {
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, chunk_out_kernel<DIM, CB>, out_smem<DIM, CB>());
    if (e != cudaSuccess) return (int)e;
    return ie_launch(chunk_out_kernel<DIM, CB>, dim3(t.chunks, t.heads, (t.vdim + CB - 1) / CB), dim3(THREADS),
                     out_smem<DIM, CB>(), t.s, t.q, t.q_ld, t.a, t.a_ld, t.w, t.w_ld, t.gates, t.gate_stride, u, u_ld, own, before, ones, t.slots, t.cu_q,
                     t.num_seqs, t.out, t.heads, t.heads_per_unit, t.dim, t.vdim, t.cols, t.q_scale, t.num_slots);
}

template <int DIM, int CB>
int launch_chunks(const Args& t, float* scratch) {
    const size_t places = (size_t)t.chunks * t.heads;
    float* add = scratch;
    float* fade = add + places * t.dim * t.vdim;
    float* ones = fade + places * t.dim;
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, chunk_state_kernel<DIM, CB>, state_smem(DIM, CB));
    if (e != cudaSuccess) return (int)e;
    int rc = ie_launch(chunk_state_kernel<DIM, CB>, dim3(t.chunks, t.heads, (t.vdim + CB - 1) / CB), dim3(THREADS),
                       state_smem(DIM, CB), t.s, t.a, t.a_ld, t.w, t.w_ld, t.gates, t.gate_stride, t.v, t.v_ld, t.cu_q, t.num_seqs,
                       t.heads, t.heads_per_unit, t.dim, t.vdim, t.cols, add, fade, ones);
    if (rc != 0) return rc;
    const int tiles = ((t.dim + 7) / 8) * ((t.vdim + 15) / 16), warps = THREADS / 32;
    rc = ie_launch(chunk_scan_kernel, dim3((tiles + warps - 1) / warps + (t.cols > t.vdim ? 1 : 0), t.heads, t.num_seqs),
                   dim3(THREADS), 0, t.s, add, (const float*)fade, ones, t.state, t.state_stride, t.slots, t.cu_q, t.heads, t.dim,
                   t.vdim, t.cols, t.num_slots);
    if (rc != 0) return rc;
    return launch_out<DIM, CB>(t, t.v, t.v_ld, 0, add, ones);
}

template <int DIM>
int launch_delta(const Args& t, const float* beta, int kv_heads, float* scratch) {
    const size_t places = (size_t)t.chunks * t.heads;
    float* U = scratch;
    float* WR = U + places * CHUNK * t.vdim;
    float* before = WR + places * wr_floats<DIM>();
    static IePerDevice allowed_solve, allowed_chain;
    cudaError_t e = ie_allow_smem(allowed_solve, delta_solve_kernel<DIM>, solve_smem<DIM>());
    if (e == cudaSuccess) e = ie_allow_smem(allowed_chain, delta_chain_kernel<DIM>, chain_smem<DIM>());
    if (e != cudaSuccess) return (int)e;
    int rc = ie_launch(delta_solve_kernel<DIM>, dim3(t.chunks, t.heads), dim3(THREADS), solve_smem<DIM>(), t.s, t.w, t.v, beta, t.a, t.cu_q,
                       t.num_seqs, t.heads, kv_heads, t.dim, t.vdim, U, WR);
    if (rc != 0) return rc;
    rc = ie_launch(delta_chain_kernel<DIM>, dim3((t.vdim + CO - 1) / CO, t.heads, t.num_seqs), dim3(THREADS), chain_smem<DIM>(), t.s, U,
                   (const float*)WR, before, t.state, t.state_stride, t.slots, t.cu_q, t.heads,
                   t.dim, t.vdim, t.num_slots);
    if (rc != 0) return rc;
    if (wide_blocks(t)) return launch_out<DIM, 128>(t, U, 0, 1, before, nullptr);
    return launch_out<DIM, 64>(t, U, 0, 1, before, nullptr);
}
}  // namespace

// Whether the kernels take these sizes: rows of whole 16-byte pieces (the caller sees to their alignment).
IE_API int ie_chunked_ok(int dim, int vdim, int delta) {
    return dim >= 4 && dim <= 128 && dim % 4 == 0 && vdim >= 4 && vdim % 4 == 0 && (!delta || vdim <= 128);
}

// Floats of scratch for so many chunks (every request's tokens of the step in chunks of 64).
IE_API long long ie_chunked_scratch(int chunks, int heads, int dim, int vdim, int delta) {
    const long long places = (long long)chunks * heads;
    const int DIM = dim > 64 ? 128 : 64;
    if (!delta) return places * ((long long)dim * vdim + 2 * dim);
    return places * ((long long)CHUNK * vdim + (DIM == 128 ? wr_floats<128>() : wr_floats<64>()) + (long long)dim * vdim);
}

// The arguments of ie_gated_recurrence, and the chunks of the step's requests (or more) with their scratch.
IE_API int ie_chunked_recurrence(const float* q, int q_ld, const float* a, int a_ld, const float* w, int w_ld,
                                 const float* gates, int gate_stride, const float* v, int v_ld, float* state,
                                 long long state_stride, const int* slots, const int* cu_q, float* out, int num_seqs, int heads,
                                 int heads_per_unit, int dim, int vdim, int cols, float q_scale, int num_slots, int chunks,
                                 float* scratch, void* stream) {
    if (num_seqs <= 0 || chunks <= 0) return 0;
    if (heads_per_unit < 1 || heads % heads_per_unit || !ie_chunked_ok(dim, vdim, 0) || q_ld % 4 || a_ld % 4 || w_ld % 4 || v_ld % 4)
        return (int)cudaErrorInvalidValue;
    if (cols < vdim || cols > vdim + 1 || (gates == nullptr && (a == nullptr || cols != vdim))) return (int)cudaErrorInvalidValue;
    Args t{q, a, w, gates, v, q_ld, a_ld, w_ld, gate_stride, v_ld, state, state_stride, slots, cu_q, out,
           num_seqs, heads, heads_per_unit, dim, vdim, cols, q_scale, num_slots, chunks, (cudaStream_t)stream};
    if (gates != nullptr) { t.a = nullptr; t.a_ld = 0; }
    if (dim > 64) return wide_blocks(t) ? launch_chunks<128, 128>(t, scratch) : launch_chunks<128, 64>(t, scratch);
    return wide_blocks(t) ? launch_chunks<64, 128>(t, scratch) : launch_chunks<64, 64>(t, scratch);
}

// The arguments of ie_delta_rule, likewise.
IE_API int ie_chunked_delta(const float* q, const float* k, const float* v, const float* beta, const float* decay, float* state,
                            long long state_stride, const int* slots, const int* cu_q, float* out, int num_seqs, int heads,
                            int kv_heads, int dim, int vdim, int num_slots, int chunks, float* scratch, void* stream) {
    if (num_seqs <= 0 || chunks <= 0) return 0;
    if (kv_heads < 1 || heads % kv_heads || !ie_chunked_ok(dim, vdim, 1)) return (int)cudaErrorInvalidValue;
    Args t{q, decay, k, nullptr, v, kv_heads * dim, heads * dim, kv_heads * dim, 0, 0, state, state_stride, slots, cu_q, out,
           num_seqs, heads, heads / kv_heads, dim, vdim, vdim, 1.0f, num_slots, chunks, (cudaStream_t)stream};
    return dim > 64 ? launch_delta<128>(t, beta, kv_heads, scratch) : launch_delta<64>(t, beta, kv_heads, scratch);
}
