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
//  * delta_solve: both right-hand sides by forward substitution, a column per thread: U = X v, W = X (p k).
//  * delta_chain: u = U - W S0 and the state after, chunk after chunk; columns of S do not interact, so a block takes 16
//    columns of a head; the next chunk's W and decayed keys are on their way meanwhile.
//  * chunk_out with those u.
//
// What bounds it: multiply-adds of the FMA pipe (40 thousand per token and head of 128 x 128), 32-bit, since a state in
// 32 bits must not lose precision to the tensor cores' 16.
#include "common.cuh"

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

// Rows that many threads read at once in a different row each lie with their 16-byte pieces turned by the row's number.
template <int DIM> __device__ __forceinline__ int turned(int row, int piece) { return row * DIM + ((piece ^ (row & 7)) << 2); }

// 64 rows of `dim` entries `ld` apart into [64][DIM], zeros beyond the chunk's rows and beyond dim.
template <int DIM, bool TURN>
__device__ __forceinline__ void fetch_rows(float* dst, const float* src, size_t ld, int cnt, int dim) {
#pragma unroll
    for (int i = threadIdx.x; i < CHUNK * DIM / 4; i += THREADS) {
        int row = i / (DIM / 4), piece = i % (DIM / 4);
        bool there = row < cnt && piece * 4 < dim;
        cp16(dst + (TURN ? turned<DIM>(row, piece) : row * DIM + piece * 4), there ? src + row * ld + piece * 4 : src, there);
    }
}

// The decays of the chunk's tokens as [64][DIM], ones beyond the chunk.  gates: one number per token (and head).
template <int DIM>
__device__ __forceinline__ void fetch_decays(float* dst, const float* a, size_t a_ld, const float* gates, size_t gate_ld,
                                             int cnt, int dim) {
#pragma unroll 4
    for (int i = threadIdx.x; i < CHUNK * DIM / 4; i += THREADS) {
        int row = i / (DIM / 4), piece = i % (DIM / 4);
        float4 v = make_float4(1.f, 1.f, 1.f, 1.f);
        if (row < cnt) {
            if (gates != nullptr) { float g = gates[row * gate_ld]; v = make_float4(g, g, g, g); }
            else if (piece * 4 < dim) v = ld4(a + row * a_ld + piece * 4);
        }
        st4(dst + row * DIM + piece * 4, v);
    }
}

// The scores of a chunk, A(i, j) = sum_d q_i D(i, j) w_j for j <= i, into [64][64] (TRANS: as A[j][i]).  qs: [64][DIM], ws: turned,
// as: [64][DIM].  Afterwards qs holds q_i times the decays from its group's start to i, ws holds w_j times the decays from j + 1 to its
// group's end, and the groups' whole decays are at `total`, in a corner of the scores that nothing else uses.
template <int DIM, bool TRANS>
struct Scores {
    static __device__ __forceinline__ int at(int i, int j) { return TRANS ? j * CHUNK + i : i * CHUNK + j; }
    static __device__ __forceinline__ int total(int group, int d) {
        int k = group * DIM + d;
        return TRANS ? (48 + (k >> 5)) * CHUNK + (k & 31) : (k >> 5) * CHUNK + 32 + (k & 31);
    }

    static __device__ __forceinline__ void run(float* qs, float* ws, const float* as, float* A) {
        const int tid = threadIdx.x;
        // inside the groups: DIM / 4 lanes hold a row's entries and go from the row's own token back to the group's first
        constexpr int LANES = DIM / 4, ROWS = THREADS / LANES;  // 32 lanes, 8 rows at once; or 16, 16
        const int lane = tid % LANES, mine = tid / LANES;
#pragma unroll 1
        for (int pass = 0; pass < CHUNK / ROWS; ++pass) {
            const int g = pass / (GROUP / ROWS);
            const int r = ROWS == GROUP ? mine : (pass & 1) ? GROUP - 1 - mine : mine;  // (a short row and a long one per warp)
            const int base = g * GROUP, row = base + r;
            float4 qd = ld4(qs + row * DIM + lane * 4);
            float part[GROUP];
#pragma unroll
            for (int j = GROUP - 1; j >= 0; --j) {
                part[j] = 0.f;
                if (j <= r) {
                    part[j] = dot4(qd, ld4(ws + turned<DIM>(base + j, lane)), 0.f);
                    qd = mul4(qd, ld4(as + (base + j) * DIM + lane * 4));
                }
            }
            // sixteen sums over the row's lanes at once: every exchange halves what a lane still holds
            int held = GROUP;
#pragma unroll
            for (int off = LANES / 2; off > 0; off >>= 1) {
                if (held > 1) {
                    held >>= 1;
                    const bool high = lane & off;
#pragma unroll
                    for (int k = 0; k < GROUP / 2; ++k) {
                        if (k < held) {
                            float send = high ? part[k] : part[k + held], keep = high ? part[k + held] : part[k];
                            part[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                        }
                    }
                } else {
                    part[0] += __shfl_xor_sync(0xffffffffu, part[0], off);
                }
            }
            const int j = LANES == 32 ? lane >> 1 : lane;
            if ((LANES == 16 || !(lane & 1)) && j <= r) A[at(row, base + j)] = part[0];
        }
        __syncthreads();
        // running products inside the groups, a column per thread
        constexpr int PARTS = THREADS / DIM, GROUPS = CHUNK / GROUP;
        {
            const int d = tid % DIM, part = tid / DIM;
#pragma unroll 1
            for (int g = part * (GROUPS / PARTS); g < (part + 1) * (GROUPS / PARTS); ++g) {
                float av[GROUP], run = 1.f;
#pragma unroll
                for (int j = 0; j < GROUP; ++j) av[j] = as[(g * GROUP + j) * DIM + d];
#pragma unroll
                for (int j = 0; j < GROUP; ++j) {
                    run *= av[j];
                    qs[(g * GROUP + j) * DIM + d] *= run;
                }
                A[total(g, d)] = run;
                run = 1.f;
#pragma unroll
                for (int j = GROUP - 1; j >= 0; --j) {
                    ws[turned<DIM>(g * GROUP + j, d >> 2) + (d & 3)] *= run;
                    run *= av[j];
                }
            }
        }
        __syncthreads();
        // between groups: the thread's entry of each of the six 16 x 16 blocks below the diagonal
        const int tx = tid & 15, ty = tid >> 4;
        float a10 = 0.f, a20 = 0.f, a21 = 0.f, a30 = 0.f, a31 = 0.f, a32 = 0.f;
#pragma unroll 4
        for (int p = 0; p < DIM / 4; ++p) {
            float4 q1 = ld4(qs + (16 + ty) * DIM + 4 * p), q2 = ld4(qs + (32 + ty) * DIM + 4 * p), q3 = ld4(qs + (48 + ty) * DIM + 4 * p);
            float4 w0 = ld4(ws + turned<DIM>(tx, p)), w1 = ld4(ws + turned<DIM>(16 + tx, p)), w2 = ld4(ws + turned<DIM>(32 + tx, p));
            float4 t1 = ld4(A + total(1, 4 * p)), t2 = ld4(A + total(2, 4 * p));
            a10 = dot4(q1, w0, a10);
            a21 = dot4(q2, w1, a21);
            a32 = dot4(q3, w2, a32);
            a20 = dot4(mul4(q2, t1), w0, a20);
            q3 = mul4(q3, t2);
            a31 = dot4(q3, w1, a31);
            a30 = dot4(mul4(q3, t1), w0, a30);
        }
        A[at(16 + ty, tx)] = a10;
        A[at(32 + ty, tx)] = a20;
        A[at(32 + ty, 16 + tx)] = a21;
        A[at(48 + ty, tx)] = a30;
        A[at(48 + ty, 16 + tx)] = a31;
        A[at(48 + ty, 32 + tx)] = a32;
        __syncthreads();
    }
};

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
    ie_pdl_trigger();
    ie_pdl_wait();
    int seq, chunk;
    const int head = blockIdx.y, c0 = blockIdx.z * CB, tid = threadIdx.x;
    if (!find_chunk(cu_q, num_seqs, blockIdx.x, seq, chunk)) return;
    const int n0 = cu_q[seq] + chunk * CHUNK, cnt = min(CHUNK, cu_q[seq + 1] - n0);
    const size_t place = (size_t)blockIdx.x * heads + head;
    fetch_rows<CB, false>(us, v + (size_t)n0 * v_ld + head * vdim + c0, v_ld, cnt, vdim - c0);
    cp_commit();
    const float* g = gates != nullptr ? gates + (size_t)n0 * gate_stride + head * 3 : nullptr;
    if (tid < CHUNK) bs[tid] = g != nullptr && tid < cnt ? g[tid * gate_stride + 1] : 0.f;
    // w_j times the decays after j: a column per thread, DIM / 256 of the chunk's tokens
    constexpr int PARTS = THREADS / DIM, EACH = CHUNK / PARTS;
    const int d = tid % DIM, part = tid / DIM;
    const float* wp = w + (size_t)n0 * w_ld + (head / heads_per_unit) * dim + d;
    const float* ap = a + (size_t)n0 * a_ld + head * dim + d;  // (not read with gates)
    float run = 1.f;
#pragma unroll 1
    for (int j1 = (part + 1) * EACH; j1 > part * EACH; j1 -= 16) {
        float wv[16], av[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            int j = j1 - 1 - i;
            bool there = j < cnt && d < dim;
            wv[i] = there ? wp[(size_t)j * w_ld] : 0.f;
            av[i] = there ? (g != nullptr ? g[j * gate_stride] : ap[(size_t)j * a_ld]) : 1.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            ws[(j1 - 1 - i) * DIM + d] = wv[i] * run;
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
    // [DIM x 64] [64 x CB]: a thread holds ROWS consecutive channels of four columns
    constexpr int LC = CB / 4, ROWS = DIM * LC / THREADS;
    const int lc = tid % LC, r0 = (tid / LC) * ROWS;
    float acc[ROWS][4];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll 2
    for (int j = 0; j < CHUNK; ++j) {
        float4 u = ld4(us + j * CB + lc * 4);
#pragma unroll
        for (int r = 0; r < ROWS; r += 4) {
            float4 x = ld4(ws + j * DIM + r0 + r);
            const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[r + k][0] = fmaf(xv[k], u.x, acc[r + k][0]);
                acc[r + k][1] = fmaf(xv[k], u.y, acc[r + k][1]);
                acc[r + k][2] = fmaf(xv[k], u.z, acc[r + k][2]);
                acc[r + k][3] = fmaf(xv[k], u.w, acc[r + k][3]);
            }
        }
    }
    const int c = c0 + lc * 4;
    if (c >= vdim) return;
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
        if (r0 + r < dim) st4(add + (place * dim + r0 + r) * vdim + c, make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]));
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
// out: [N, heads, cols], times q_scale.  112 KB of shared memory, two blocks per SM: the state, then u, take the place of w and the
// decays once the scores stand.
template <int DIM, int CB>
__global__ void __launch_bounds__(THREADS, 2)
chunk_out_kernel(const float* __restrict__ q, int q_ld, const float* __restrict__ a, int a_ld, const float* __restrict__ w,
                 int w_ld, const float* __restrict__ gates, int gate_stride, const float* __restrict__ u, int u_ld, int own,
                 const float* __restrict__ before, const float* __restrict__ ones, const int* __restrict__ slots,
                 const int* __restrict__ cu_q, int num_seqs, float* __restrict__ out, int heads, int heads_per_unit, int dim,
                 int vdim, int cols, float q_scale, int num_slots) {
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;                // [64][DIM]
    float* ws = qs + CHUNK * DIM;  // [64][DIM], then with the next the state [DIM][CB], then u [64][CB]
    float* as = ws + CHUNK * DIM;  // [64][DIM]
    float* A = as + CHUNK * DIM;   // [64][64]
    using Sc = Scores<DIM, false>;
    ie_pdl_trigger();
    ie_pdl_wait();
    int seq, chunk;
    const int head = blockIdx.y, c0 = blockIdx.z * CB, tid = threadIdx.x, unit = head / heads_per_unit;
    if (!find_chunk(cu_q, num_seqs, blockIdx.x, seq, chunk)) return;
    const int n0 = cu_q[seq] + chunk * CHUNK, cnt = min(CHUNK, cu_q[seq + 1] - n0), slot = slots[seq];
    if (slot < 0 || slot >= num_slots) return;
    const size_t place = (size_t)blockIdx.x * heads + head;
    const float* g = gates != nullptr ? gates + (size_t)n0 * gate_stride + head * 3 : nullptr;
    fetch_rows<DIM, false>(qs, q + (size_t)n0 * q_ld + unit * dim, q_ld, cnt, dim);
    fetch_rows<DIM, true>(ws, w + (size_t)n0 * w_ld + unit * dim, w_ld, cnt, dim);
    cp_commit();
    fetch_decays<DIM>(as, a + (size_t)n0 * a_ld + head * dim, a_ld, g, gate_stride, cnt, dim);
    cp_wait<0>();
    __syncthreads();
    Sc::run(qs, ws, as, A);
    // the state comes while the queries take the decays of the groups before theirs
    float* Ss = ws;
#pragma unroll
    for (int i = tid; i < DIM * CB / 4; i += THREADS) {
        int d = i / (CB / 4), c = (i % (CB / 4)) * 4;
        bool there = d < dim && c0 + c < vdim;
        cp16(Ss + d * CB + c, there ? before + (place * dim + d) * vdim + c0 + c : before, there);
    }
    cp_commit();
    {
        constexpr int PARTS = THREADS / DIM, EACH = CHUNK / PARTS;
        const int d = tid % DIM, part = tid / DIM;
        float pre = 1.f;
        for (int grp = 0; grp < (part + 1) * EACH / GROUP; ++grp) {
            if (grp >= part * EACH / GROUP && grp > 0)
#pragma unroll
                for (int j = 0; j < GROUP; ++j) qs[(grp * GROUP + j) * DIM + d] *= pre;
            pre *= A[Sc::total(grp, d)];
        }
    }
    cp_wait<0>();
    __syncthreads();
    constexpr int LC = CB / 4, ROWS = CHUNK * LC / THREADS;  // a thread: ROWS consecutive tokens, four columns
    const int lc = tid % LC, r0 = (tid / LC) * ROWS;
    float acc[ROWS][4];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll 2
    for (int p = 0; p < DIM / 4; ++p) {
        float4 s[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] = ld4(Ss + (4 * p + k) * CB + lc * 4);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            float4 x = ld4(qs + (r0 + r) * DIM + 4 * p);
            const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[r][0] = fmaf(xv[k], s[k].x, acc[r][0]);
                acc[r][1] = fmaf(xv[k], s[k].y, acc[r][1]);
                acc[r][2] = fmaf(xv[k], s[k].z, acc[r][2]);
                acc[r][3] = fmaf(xv[k], s[k].w, acc[r][3]);
            }
        }
    }
    __syncthreads();
    float* us = ws;
    if (own) fetch_rows<CB, false>(us, u + place * CHUNK * vdim + c0, vdim, cnt, vdim - c0);
    else fetch_rows<CB, false>(us, u + (size_t)n0 * u_ld + head * vdim + c0, u_ld, cnt, vdim - c0);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    if (g != nullptr) {
        for (int i = tid; i < CHUNK * CB; i += THREADS) {
            int j = i / CB;
            us[i] *= j < cnt ? g[j * gate_stride + 1] : 0.f;
        }
        __syncthreads();
    }
    // tokens before the thread's own, then (the triangle) its own: no token reads a later one's value, whatever it is
#pragma unroll 2
    for (int p = 0; p < r0 / 4; ++p) {
        float4 s[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] = ld4(us + (4 * p + k) * CB + lc * 4);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            float4 x = ld4(A + (r0 + r) * CHUNK + 4 * p);
            const float xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[r][0] = fmaf(xv[k], s[k].x, acc[r][0]);
                acc[r][1] = fmaf(xv[k], s[k].y, acc[r][1]);
                acc[r][2] = fmaf(xv[k], s[k].z, acc[r][2]);
                acc[r][3] = fmaf(xv[k], s[k].w, acc[r][3]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        float4 s = ld4(us + (r0 + j) * CB + lc * 4);
#pragma unroll
        for (int r = j; r < ROWS; ++r) {
            float x = A[(r0 + r) * CHUNK + r0 + j];
            acc[r][0] = fmaf(x, s.x, acc[r][0]);
            acc[r][1] = fmaf(x, s.y, acc[r][1]);
            acc[r][2] = fmaf(x, s.z, acc[r][2]);
            acc[r][3] = fmaf(x, s.w, acc[r][3]);
        }
    }
    const int c = c0 + lc * 4;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (r0 + r >= cnt || c >= vdim) break;
        float* o = out + ((size_t)(n0 + r0 + r) * heads + head) * cols + c;
        if (cols == vdim) {
            st4(o, make_float4(acc[r][0] * q_scale, acc[r][1] * q_scale, acc[r][2] * q_scale, acc[r][3] * q_scale));
        } else {  // (rows of an odd length)
#pragma unroll
            for (int k = 0; k < 4; ++k) o[k] = acc[r][k] * q_scale;
        }
    }
    if (cols > vdim && c0 == 0) {  // the normaliser's column, whose values are the gates
        const int warp = tid >> 5, lane = tid & 31;
        for (int i = warp; i < cnt; i += THREADS / 32) {
            float s = 0.f;
            for (int d = lane; d < dim; d += 32) s = fmaf(qs[i * DIM + d], ones[place * dim + d], s);
            for (int j = lane; j <= i; j += 32) s = fmaf(A[i * CHUNK + j], g[j * gate_stride + 1], s);
            s = warp_sum(s);
            if (lane == 0) out[((size_t)(n0 + i) * heads + head) * cols + vdim] = s * q_scale;
        }
    }
}

// grid: (chunks, heads).  U: [chunks, heads, 64, vdim]; W: [chunks, heads, 64, DIM] with the pieces of 16 bytes turned by the row's
// number; R: [chunks, heads, 64, DIM], the keys times the decays after them; fade: [chunks, heads, DIM].
template <int DIM>
__global__ void __launch_bounds__(THREADS, 2)
delta_solve_kernel(const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ beta,
                   const float* __restrict__ decay, const int* __restrict__ cu_q, int num_seqs, int heads, int kv_heads,
                   int dim, int vdim, float* __restrict__ U, float* __restrict__ W, float* __restrict__ R,
                   float* __restrict__ fade) {
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;
    float* ws = qs + CHUNK * DIM;
    float* as = ws + CHUNK * DIM;
    float* Lt = as + CHUNK * DIM;  // [j][i]
    using Sc = Scores<DIM, true>;
    auto beta_at = [](int i) { return (32 + (i >> 5)) * CHUNK + (i & 31); };  // (another corner without scores)
    ie_pdl_trigger();
    ie_pdl_wait();
    int seq, chunk;
    const int head = blockIdx.y, tid = threadIdx.x, kvh = head / (heads / kv_heads);
    if (!find_chunk(cu_q, num_seqs, blockIdx.x, seq, chunk)) return;
    const int n0 = cu_q[seq] + chunk * CHUNK, cnt = min(CHUNK, cu_q[seq + 1] - n0);
    const size_t place = (size_t)blockIdx.x * heads + head;
    const float* kp = k + ((size_t)n0 * kv_heads + kvh) * dim;
    fetch_rows<DIM, false>(qs, kp, (size_t)kv_heads * dim, cnt, dim);
    fetch_rows<DIM, true>(ws, kp, (size_t)kv_heads * dim, cnt, dim);
    cp_commit();
    fetch_decays<DIM>(as, decay + ((size_t)n0 * heads + head) * dim, (size_t)heads * dim, nullptr, 0, cnt, dim);
    if (tid < CHUNK) Lt[beta_at(tid)] = tid < cnt ? beta[(size_t)(n0 + tid) * heads + head] : 0.f;
    cp_wait<0>();
    __syncthreads();
    Sc::run(qs, ws, as, Lt);
    const bool is_key = tid < DIM;
    const int d = tid, c = tid - DIM;
    float x[CHUNK];
    if (is_key) {  // W's right-hand side; the keys that the state's update takes
        float pre = 1.f;
#pragma unroll
        for (int g = 0; g < CHUNK / GROUP; ++g) {
#pragma unroll
            for (int i = 0; i < GROUP; ++i) x[g * GROUP + i] = qs[(g * GROUP + i) * DIM + d] * pre;
            pre *= Lt[Sc::total(g, d)];
        }
        fade[place * DIM + d] = pre;
        float after = 1.f;
        float* r = R + place * CHUNK * DIM + d;
#pragma unroll 1
        for (int g = CHUNK / GROUP - 1; g >= 0; --g) {
#pragma unroll
            for (int j = 0; j < GROUP; ++j)
                r[(g * GROUP + j) * DIM] = ws[turned<DIM>(g * GROUP + j, d >> 2) + (d & 3)] * after;
            after *= Lt[Sc::total(g, d)];
        }
    } else {
        const float* vp = v + ((size_t)n0 * heads + head) * vdim + c;
#pragma unroll
        for (int i = 0; i < CHUNK; ++i) x[i] = i < cnt && c < vdim ? vp[(size_t)i * heads * vdim] : 0.f;
    }
    // rows times beta, on both sides
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) x[i] *= Lt[beta_at(i)];
    __syncthreads();
    for (int i = tid; i < CHUNK * CHUNK; i += THREADS) {
        int j = i / CHUNK, row = i % CHUNK;
        if (row > j) Lt[i] *= Lt[beta_at(row)];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < CHUNK - 1; ++j) {
#pragma unroll
        for (int p = (j + 1) / 4; p < CHUNK / 4; ++p) {
            float4 l = ld4(Lt + j * CHUNK + 4 * p);
            const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (4 * p + i > j) x[4 * p + i] = fmaf(-lv[i], x[j], x[4 * p + i]);
        }
    }
    if (is_key) {
        float* out = W + place * CHUNK * DIM;
#pragma unroll
        for (int i = 0; i < CHUNK; ++i) out[turned<DIM>(i, d >> 2) + (d & 3)] = x[i];
    } else if (c < vdim) {
        float* out = U + place * CHUNK * vdim + c;
#pragma unroll
        for (int i = 0; i < CHUNK; ++i) out[i * vdim] = x[i];
    }
}

// grid: (blocks of 16 columns, heads, requests).  U becomes u; before: [chunks, heads, dim, vdim].
// Shared memory is what bounds it (a row of W serves sixteen columns only), so every access of W and R is of 512 different bytes and the
// state and u come as one value for the whole warp.  u = U - W S0: a warp takes an eighth of the channels, a lane two rows of W with all
// sixteen columns.  The state: a warp takes a quarter of the tokens (dim 64: an eighth) and eight columns, a lane four channels.  The
// warps' sums meet in shared memory in a fixed order.
constexpr int CO = 16, RED_LD = CHUNK + 2, CHAIN_RED = 8 * CO * RED_LD;
template <int DIM>
__global__ void __launch_bounds__(THREADS)
delta_chain_kernel(float* __restrict__ U, const float* __restrict__ W, const float* __restrict__ R, const float* __restrict__ fade,
                   float* __restrict__ before, float* __restrict__ state, long long state_stride, const int* __restrict__ slots,
                   const int* __restrict__ cu_q, int heads, int dim, int vdim, int num_slots) {
    extern __shared__ __align__(16) float sm[];
    constexpr int TILE = CHUNK * DIM, LD = DIM + 4;
    float* Wb = sm;                // two of [64][DIM]
    float* Rb = Wb + 2 * TILE;     // two of [64][DIM]
    float* red = Rb + 2 * TILE;    // CHAIN_RED floats
    float* Ss = red + CHAIN_RED;   // [16][LD]
    float* Us = Ss + CO * LD;      // [64][16]
    float* Ps = Us + CHUNK * CO;   // two of [DIM]
    ie_pdl_trigger();
    ie_pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z, c0 = blockIdx.x * CO, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int len = cu_q[seq + 1] - cu_q[seq], slot = slots[seq];
    if (len <= 0 || slot < 0 || slot >= num_slots) return;
    int first = 0;
    for (int s = 0; s < seq; ++s) first += (cu_q[s + 1] - cu_q[s] + CHUNK - 1) / CHUNK;
    const int chunks = (len + CHUNK - 1) / CHUNK;
    float* S = state + (size_t)slot * state_stride + ((size_t)head * vdim + c0) * dim;
    for (int i = tid; i < CO * DIM; i += THREADS) {
        int c = i / DIM, d = i % DIM;
        Ss[c * LD + d] = c0 + c < vdim && d < dim ? S[(size_t)c * dim + d] : 0.f;
    }
    auto fetch = [&](int c, int b) {
        const size_t place = (size_t)(first + c) * heads + head;
#pragma unroll
        for (int i = tid; i < TILE / 4; i += THREADS) {
            cp16(Wb + b * TILE + 4 * i, W + place * TILE + 4 * i, true);
            cp16(Rb + b * TILE + 4 * i, R + place * TILE + 4 * i, true);
        }
        if (tid < DIM / 4) cp16(Ps + b * DIM + 4 * tid, fade + place * DIM + 4 * tid, true);
    };
    fetch(0, 0);
    cp_commit();
    const int urow = tid >> 2, ucol = (tid & 3) * 4;  // the thread's four of u when the warps' sums meet
    const bool ucols = c0 + ucol < vdim;
    for (int c = 0; c < chunks; ++c) {
        const int b = c & 1;
        const size_t place = (size_t)(first + c) * heads + head;
        float* up = U + (place * CHUNK + urow) * vdim + c0 + ucol;
        float4 mine = ucols ? ld4(up) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (c + 1 < chunks) fetch(c + 1, b ^ 1);
        cp_commit();
        cp_wait<1>();
        __syncthreads();
        // the state before the chunk, for the outputs
#pragma unroll
        for (int i = tid; i < DIM * CO / 4; i += THREADS) {
            int d = i >> 2, cc = (i & 3) * 4;
            if (d < dim && c0 + cc < vdim)
                st4(before + (place * dim + d) * vdim + c0 + cc,
                    make_float4(Ss[cc * LD + d], Ss[(cc + 1) * LD + d], Ss[(cc + 2) * LD + d], Ss[(cc + 3) * LD + d]));
        }
        {
            float acc[2][CO];
#pragma unroll
            for (int i = 0; i < CO; ++i) acc[0][i] = acc[1][i] = 0.f;
            const float* w0 = Wb + b * TILE + lane * DIM;
            const int turn = lane & 7;
#pragma unroll 2
            for (int p = warp * (DIM / 32); p < (warp + 1) * (DIM / 32); ++p) {
                float4 x0 = ld4(w0 + ((p ^ turn) << 2)), x1 = ld4(w0 + 32 * DIM + ((p ^ turn) << 2));
#pragma unroll
                for (int cc = 0; cc < CO; ++cc) {
                    float4 s = ld4(Ss + cc * LD + 4 * p);
                    acc[0][cc] = dot4(x0, s, acc[0][cc]);
                    acc[1][cc] = dot4(x1, s, acc[1][cc]);
                }
            }
            // [8 warps][16 columns][64 rows and two]
            float* p = red + warp * (CO * RED_LD) + lane;
#pragma unroll
            for (int cc = 0; cc < CO; ++cc) {
                p[cc * RED_LD] = acc[0][cc];
                p[cc * RED_LD + 32] = acc[1][cc];
            }
        }
        __syncthreads();
        {
            float s[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float t = 0.f;
#pragma unroll
                for (int w = 0; w < 8; ++w) t += red[(w * CO + ucol + i) * RED_LD + urow];
                s[i] = t;
            }
            mine = make_float4(mine.x - s[0], mine.y - s[1], mine.z - s[2], mine.w - s[3]);
            st4(Us + urow * CO + ucol, mine);
            if (ucols) st4(up, mine);
        }
        __syncthreads();
        constexpr int LANES = DIM / 4, KS = THREADS / LANES / 2, TOKENS = CHUNK / KS;  // lanes of a row; shares of the tokens
        {
            const int sub = tid % LANES, group = tid / LANES, half = (group & 1) * 8, ks = group >> 1;
            float acc[4][8];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[r][i] = 0.f;
            const float* rt = Rb + b * TILE + sub * 4;
#pragma unroll 4
            for (int j = ks * TOKENS; j < (ks + 1) * TOKENS; ++j) {
                float4 x = ld4(rt + j * DIM), y0 = ld4(Us + j * CO + half), y1 = ld4(Us + j * CO + half + 4);
                const float xv[4] = {x.x, x.y, x.z, x.w}, yv[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[r][i] = fmaf(xv[r], yv[i], acc[r][i]);
            }
            // [KS][16 columns][DIM]
#pragma unroll
            for (int i = 0; i < 8; ++i)
                st4(red + (ks * CO + half + i) * DIM + sub * 4, make_float4(acc[0][i], acc[1][i], acc[2][i], acc[3][i]));
        }
        __syncthreads();
#pragma unroll
        for (int i = tid; i < CO * DIM / 4; i += THREADS) {
            int cc = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
            float4 s = ld4(Ss + cc * LD + d), f = ld4(Ps + b * DIM + d), t = ld4(red + cc * DIM + d);
#pragma unroll
            for (int j = 1; j < KS; ++j) {
                float4 n = ld4(red + (j * CO + cc) * DIM + d);
                t = make_float4(t.x + n.x, t.y + n.y, t.z + n.z, t.w + n.w);
            }
            st4(Ss + cc * LD + d, make_float4(fmaf(f.x, s.x, t.x), fmaf(f.y, s.y, t.y), fmaf(f.z, s.z, t.z), fmaf(f.w, s.w, t.w)));
        }
        __syncthreads();
    }
    for (int i = tid; i < CO * DIM; i += THREADS) {
        int c = i / DIM, d = i % DIM;
        if (c0 + c < vdim && d < dim) S[(size_t)c * dim + d] = Ss[c * LD + d];
    }
}

constexpr size_t out_smem(int dim) { return (size_t)(3 * CHUNK * dim + CHUNK * CHUNK) * sizeof(float); }
constexpr size_t state_smem(int dim, int cb) { return (size_t)(CHUNK * (dim + cb) + THREADS + CHUNK) * sizeof(float); }
constexpr size_t chain_smem(int dim) { return (size_t)(4 * CHUNK * dim + CHAIN_RED + CO * (dim + 4) + CHUNK * CO + 2 * dim) * sizeof(float); }

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
    cudaError_t e = ie_allow_smem(allowed, chunk_out_kernel<DIM, CB>, out_smem(DIM));
    if (e != cudaSuccess) return (int)e;
    return ie_launch(chunk_out_kernel<DIM, CB>, dim3(t.chunks, t.heads, (t.vdim + CB - 1) / CB), dim3(THREADS), out_smem(DIM), t.s,
                     t.q, t.q_ld, t.a, t.a_ld, t.w, t.w_ld, t.gates, t.gate_stride, u, u_ld, own, before, ones, t.slots, t.cu_q,
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
    float* W = U + places * CHUNK * t.vdim;
    float* R = W + places * CHUNK * DIM;
    float* before = R + places * CHUNK * DIM;
    float* fade = before + places * t.dim * t.vdim;
    static IePerDevice allowed_solve, allowed_chain;
    cudaError_t e = ie_allow_smem(allowed_solve, delta_solve_kernel<DIM>, out_smem(DIM));
    if (e == cudaSuccess) e = ie_allow_smem(allowed_chain, delta_chain_kernel<DIM>, chain_smem(DIM));
    if (e != cudaSuccess) return (int)e;
    int rc = ie_launch(delta_solve_kernel<DIM>, dim3(t.chunks, t.heads), dim3(THREADS), out_smem(DIM), t.s, t.w, t.v, beta, t.a, t.cu_q,
                       t.num_seqs, t.heads, kv_heads, t.dim, t.vdim, U, W, R, fade);
    if (rc != 0) return rc;
    rc = ie_launch(delta_chain_kernel<DIM>, dim3((t.vdim + CO - 1) / CO, t.heads, t.num_seqs), dim3(THREADS), chain_smem(DIM), t.s, U,
                   (const float*)W, (const float*)R, (const float*)fade, before, t.state, t.state_stride, t.slots, t.cu_q, t.heads,
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
    return places * ((long long)CHUNK * vdim + 2 * CHUNK * DIM + (long long)dim * vdim + DIM);
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
