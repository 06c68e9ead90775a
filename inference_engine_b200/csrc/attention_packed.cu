// Softmax attention of prompt portions on the fifth-generation tensor cores, bfloat16, with what the engine's softmax mixers ask
// for: a sink, a sliding window beside kept first positions, capped scores, an output gate.  Built per (key size PA_D: 64, 128 or 192;
// value size PA_DV: 64 or 128).
//
// A block owns 256 rows of one request and one key/value head, a row being a (token, query head of the group) pair, so that a key tile
// is brought once for the whole group, and walks tiles of 64 keys.  Two row tiles of 128 take turns, and a row tile's scores are made a key tile
// ahead of its softmax, so that softmax follows softmax.  Twelve warps (a thirteenth would leave a thread 128 registers instead of
// 168, and it would spill):
//   warps 0-3, 4-7: softmax of row tile 0 and 1, a thread per row (tensor-memory lane);
//   warps 8, 9: tcgen05.mma of row tile 0 and 1.  Per key tile: O += P V as the weights are written (P in tensor memory, over the scores it
//     was made from), then S = Q K^T of the key tile after the next (both operands from shared memory);
//   warps 10, 11: gather keys and values by cp.async, every other key tile each, swizzled by hand as the tensor core reads them.  (Pages of
//     16 tokens as TMA boxes are 2 KB each, and the copy engine spends 120 to 300 clocks on any box: they would take longer than a tile's
//     products.)
// Tensor memory: row tile i's scores of key tile t in columns (2 i + t % 2) 64 .. + 63, its output in 256 + 128 i.  A row's weights replace its
// scores: 32 columns of weights rounded to bfloat16, two to a column, then 32 columns of what the rounding left (a weight keeps 16 bits of
// mantissa; both go through the second product).  The maximum that weights are taken against follows a row's running maximum only when that
// has grown by more than 2^8; only then is the row's output rescaled.  A row's arithmetic depends on its own request alone.
//
// PA_FLAT 1 (latent attention whose keys and values were expanded per head): keys and values are rows of step-wide arrays, a request's
// context after the one before it; a key is the head's own entries (PA_D - 64) and then up to 64 rotated ones that all heads share.
//
// What bounds it: a key tile's products take 1,840 clocks with two terms and keys of 128 (65 for 128 x 128 x 16, 50 for 128 x 64 x 16, as
// measured), its exponentials 1,024 of the special-function unit; a tile takes 1,940.  Keys of 64: 1,880, softmax and the way round (weights,
// product, scores) about as long as each other.  What it was before: scores one tile of 128 keys at a time, made when the softmax before
// had ended, 7,000 per 128 keys; a tile ahead, with copies fenced by the warps that all shared a tile, 2,700.
// Sixteen query heads on four of 128: window 1,024, 2,048 tokens 31 us (the mma.sync kernel that serves the other sizes: 142);
// 8,192 tokens, all positions, 280 us.
//
// PA_PROMPT: plain attention as Llama-like models have it.  One term of the weights (as the kernel of 128 tokens of a head a block has
// it), all portions of a step in one grid, and the key tiles of a block's rows cut among a cluster of blocks, whose outputs are added through
// the cluster's shared memory (through scratch by the block that ended last it took 8 us for 9 parts).  Softmax bounds it: 1,500 clocks a tile
// with keys of 64, 1,650 with 128 (products 600 and 1,320).  Against the kernel of a head a block, 32 heads on 8, us: 2,048 tokens of 128
// entries 85 -> 42, 8,192 tokens 849 -> 449, 512 tokens behind 8,192 118 -> 78; of 64 entries 39 -> 35, 424 -> 374, 68 -> 65.
// Every wait is bounded; a block that waits too long records IE_ERR_TIMEOUT, frees its tensor memory and leaves.
#include "tma.cuh"
#include <math.h>

#ifndef PA_D
#define PA_D 128
#endif
#ifndef PA_DV
#define PA_DV 128
#endif
#ifndef PA_FLAT
#define PA_FLAT 0
#endif
#ifndef PA_PROMPT
#define PA_PROMPT 0
#endif

using namespace ie_tma;

namespace {
constexpr int D = PA_D, DV = PA_DV;
static_assert((D == 64 || D == 128 || D == 192) && (DV == 64 || DV == 128), "sizes");
constexpr bool FLAT = PA_FLAT != 0;
constexpr bool PROMPT = PA_PROMPT != 0;
static_assert(!(FLAT && PROMPT), "one form at a time");
constexpr int TERMS = PROMPT ? 1 : 2;
constexpr int BM = 128, ROWS = 2 * BM, KT = 64;
constexpr int KH = D / 64, VH = DV / 64;         // runs of 64 entries: 128 bytes, one swizzle atom
constexpr int Q_RUN = BM * 128, KV_RUN = KT * 128;  // such a run of a row tile, of a key tile
constexpr int K_BYTES = KH * KV_RUN, V_BYTES = VH * KV_RUN, Q_TILE = KH * Q_RUN, Q_BYTES = 2 * Q_TILE;
constexpr int KS = D == 192 ? 3 : 4, VS = D == 192 ? 3 : 4;  // tiles of keys and of values in shared memory
constexpr int SOFTMAX_WARPS = 8, MMA_WARPS = 2, COPY_WARPS = 2, THREADS = (SOFTMAX_WARPS + MMA_WARPS + COPY_WARPS) * 32;
constexpr float RESCALE_LAG = 8.0f;              // in powers of two
constexpr float LOG2E_F = 1.4426950408889634f;

struct __align__(8) Bars {
    unsigned long long q_full, k_full[KS], k_empty[KS], v_full[VS], v_empty[VS], s_done[4], p_ready[4], o_done[2];
    unsigned tmem_base;
    int failed;
};
constexpr int MOST_SHARES = 8;  // blocks of a cluster that every device runs
static_assert(ROWS * (DV * 4 + 8) <= Q_BYTES + KS * K_BYTES + VS * V_BYTES, "room for the shares");
constexpr size_t SMEM_BYTES = (size_t)Q_BYTES + KS * K_BYTES + VS * V_BYTES + sizeof(Bars) + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

// Shared-memory descriptors as their two words: the low one (start address and, for values, the distance of the runs, in 16-byte units)
// moves with the address, the high one (groups of eight rows 1,024 bytes apart, version, 128-byte swizzle) is a constant.  An instruction
// then costs an addition an operand; descriptors put together anew for each cost the issuing warp 100 clocks an instruction beside
// the softmax warps, where the tensor core needs 48 and 65.
constexpr unsigned DESC_HIGH = (1024u >> 4) | (1u << 14) | (2u << 29);
// (within a cluster an address has the block's number above its 18 bits)
__device__ __forceinline__ unsigned desc_low(unsigned addr, unsigned run) { return ((addr & 0x3ffff) >> 4) | ((run >> 4) << 16); }
__device__ __forceinline__ void mma_ss(unsigned d, unsigned a, unsigned b, unsigned idesc, bool accumulate) {
    asm volatile("{\n .reg .pred p;\n .reg .b64 x, y;\n setp.ne.b32 p, %5, 0;\n mov.b64 x, {%1, %3};\n mov.b64 y, {%2, %3};\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %4, p;\n}"
                 ::"r"(d), "r"(a), "r"(b), "r"(DESC_HIGH), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
__device__ __forceinline__ void mma_ts(unsigned d, unsigned a, unsigned b, unsigned idesc, bool accumulate) {
    asm volatile("{\n .reg .pred p;\n .reg .b64 y;\n setp.ne.b32 p, %5, 0;\n mov.b64 y, {%2, %3};\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], y, %4, p;\n}"
                 ::"r"(d), "r"(a), "r"(b), "r"(DESC_HIGH), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
__device__ __forceinline__ void cp16(unsigned dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// tanh from one exponential: 1 - 2 / (e^(2x) + 1), the argument held where tanh is 1 to 32-bit precision
__device__ __forceinline__ float tanh_fast(float x) {
    x = fminf(fmaxf(x, -15.f), 15.f);
    return 1.f - __fdividef(2.f, __expf(2.f * x) + 1.f);
}
__device__ __forceinline__ float2 as_float2(unsigned packed) {  // two bfloat16 as 32-bit numbers
    return make_float2(__uint_as_float(packed << 16), __uint_as_float(packed & 0xffff0000u));
}
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}

// 16 columns of this thread's lane (the caller waits for the stores).
__device__ __forceinline__ void tmem_st16(const unsigned (&r)[16], unsigned taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}

struct Inputs {
    const bf16 *q, *k, *v;  // q: [tokens, heads, D]; k, v: the paged caches
    const int *tables, *cu_q, *ctx_lens;
    int table_width, heads, kv_heads, page_shift, total_pages;
    float scale;
    int window, keep_first;
    float softcap;
    const float *sinks, *gate;  // gate: per head at [token * gate_ld + head], or per value entry (gate_elements)
    int gate_ld, gate_elements;
    bf16* out;
    int out_ld;
    // PA_FLAT: q [tokens, heads, D - 64], the rotated entries of (token, head) at q_rot + (token * heads + head) * q_rot_ld; keys and
    // values at k + row * kv_ld + head * (D - 64) and v + row * kv_ld + head * DV, the shared rotated entries (`rot` of them) at k_rot + row *
    // k_rot_ld
    const bf16 *q_rot, *k_rot;
    int q_rot_ld, k_rot_ld, kv_ld, rot;
    // PA_PROMPT: the step's requests (those of 16 rows or fewer are another kernel's)
    int num_seqs;
};

__device__ __forceinline__ unsigned peer_smem(unsigned addr, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A cluster's blocks hold 256 rows' shares of the output (relative to the share's maximum; piece c of 16 bytes of row r in place c ^ (r & 7)), maxima
// and sums in shared memory, and each adds an even part of the rows, in the order of the shares.  DV / 4 lanes take a row; a lane works one
// share's factor out.
__device__ __forceinline__ void add_shares(unsigned o_s, unsigned ml_s, int rank, int shares, bf16* out, int out_ld, int row0, int rows_here,
                                           int group, int tid) {
    constexpr int LANES = DV / 4, AT_ONCE = THREADS / LANES;
    const int c = tid % LANES, end = (rank + 1) * rows_here / shares;
    for (int r1 = rank * rows_here / shares; r1 < end; r1 += AT_ONCE) {
        const int r = min(r1 + tid / LANES, end - 1);
        float m = -INFINITY, l = 0.f;
        if (c < shares) asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(m), "=f"(l) : "r"(peer_smem(ml_s + r * 8, c)));
        float4 v[MOST_SHARES];
#pragma unroll
        for (int z = 0; z < MOST_SHARES; ++z)
            if (z < shares)
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[z].x), "=f"(v[z].y), "=f"(v[z].z), "=f"(v[z].w)
                             : "r"(peer_smem(o_s + r * (DV * 4) + ((c ^ (r & 7)) << 4), z)));
        float top = m;
#pragma unroll
        for (int x = 1; x < MOST_SHARES; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x, LANES));
        top = __shfl_sync(0xffffffffu, top, 0, LANES);
        float f = m == -INFINITY ? 0.f : fast_exp2(m - top);
        float sum = l * f;
#pragma unroll
        for (int x = 1; x < MOST_SHARES; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x, LANES);
        sum = __shfl_sync(0xffffffffu, sum, 0, LANES);
        f *= sum > 0.f ? 1.f / sum : 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int z = 0; z < MOST_SHARES; ++z) {
            if (z >= shares) break;
            const float g = __shfl_sync(0xffffffffu, f, z, LANES);
            acc.x = fmaf(v[z].x, g, acc.x); acc.y = fmaf(v[z].y, g, acc.y); acc.z = fmaf(v[z].z, g, acc.z); acc.w = fmaf(v[z].w, g, acc.w);
        }
        if (r1 + tid / LANES < end) {
            const int rr = row0 + r, token = rr / group;
            *reinterpret_cast<uint2*>(out + (size_t)token * out_ld + (rr - token * group) * DV + c * 4) = make_uint2(pack2(acc.x, acc.y), pack2(acc.z, acc.w));
        }
    }
}

// grid: (blocks of 256 rows of the longest portion x key/value heads, requests): the rows that see most start first, whatever the head
// (PA_PROMPT: (blocks of 256 rows of all portions x key/value heads, shares): SHARED, a cluster of blocks takes a block's key tiles)
template <bool CAP, bool SHARED>
__global__ void __launch_bounds__(THREADS, 1)
attention_packed_kernel(const Inputs in, int* err) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* q_s = smem;                      // [row tile][run][128 rows][128 bytes]
    unsigned char* k_s = q_s + Q_BYTES;             // [slot][run][128 keys][128 bytes]
    unsigned char* v_s = k_s + KS * K_BYTES;
    Bars* bars = reinterpret_cast<Bars*>(v_s + VS * V_BYTES);
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (one number for the whole warp, as far as the compiler is concerned)
    ie_pdl_trigger();
    // (lengths and block tables are the step's inputs; queries, keys and values are the kernels' before)
    const int kvh = blockIdx.x % in.kv_heads, group = in.heads / in.kv_heads;
    int block = (gridDim.x - 1 - blockIdx.x) / in.kv_heads, seq = PROMPT ? -1 : (int)blockIdx.y;
    if (PROMPT) {  // the grid's blocks are the requests' one after the other
        for (int i = 0; i < in.num_seqs; ++i) {
            const int rows = (in.cu_q[i + 1] - in.cu_q[i]) * group, blocks = rows > 16 ? (rows + ROWS - 1) / ROWS : 0;
            if (block < blocks) { seq = i; break; }
            block -= blocks;
        }
        if (seq < 0) { ie_pdl_leave(); return; }
    }
    const int q0 = in.cu_q[seq], q_len = in.cu_q[seq + 1] - q0;
    const int row0 = block * ROWS, rows_total = q_len * group;
    if (row0 >= rows_total) { ie_pdl_leave(); return; }
    const int start = in.ctx_lens[seq] - q_len;  // position of the request's first token of this step
    const int rows_here = min(ROWS, rows_total - row0);
    const int first_pos = start + row0 / group, last_pos = start + (row0 + rows_here - 1) / group;
    const int lo_min = in.window > 0 ? max(first_pos - in.window + 1, 0) : 0;
    // the tiles the block walks, by a running number: those that hold kept keys and lie before the window's first, then the window's
    const int win_begin = lo_min / KT, win_end = last_pos / KT;
    const int kept_tiles = in.keep_first > 0 ? min((in.keep_first - 1) / KT + 1, win_begin) : 0;
    const int all_tiles = kept_tiles + win_end - win_begin + 1;
    const int shares = SHARED ? (int)gridDim.y : 1, share = SHARED ? (int)blockIdx.y : 0;  // (a share may be empty)
    const int tile0 = share * all_tiles / shares, tiles = (share + 1) * all_tiles / shares - tile0;
    auto key_of = [&](int t) { t += tile0; return (t < kept_tiles ? t : win_begin + t - kept_tiles) * KT; };
    const int row_tiles = rows_here > BM ? 2 : 1;  // (a second one without rows is left out)

    if (tid == 0) {
        mbar_init(&bars->q_full, SOFTMAX_WARPS);
        for (int s = 0; s < KS; ++s) { mbar_init(&bars->k_full[s], 1); mbar_init(&bars->k_empty[s], row_tiles); }
        for (int s = 0; s < VS; ++s) { mbar_init(&bars->v_full[s], 1); mbar_init(&bars->v_empty[s], row_tiles); }
        for (int i = 0; i < 4; ++i) { mbar_init(&bars->s_done[i], 1); mbar_init(&bars->p_ready[i], BM); }
        for (int i = 0; i < 2; ++i) mbar_init(&bars->o_done[i], 1);
        bars->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == SOFTMAX_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = __shfl_sync(0xffffffffu, bars->tmem_base, 0);
    ie_pdl_wait();

    if (warp >= SOFTMAX_WARPS && warp < SOFTMAX_WARPS + MMA_WARPS) {
        // ---- tensor core: a warp per row tile ----
        const int i = warp - SOFTMAX_WARPS;
        const unsigned idesc_qk = umma_idesc_bf16(BM, KT), idesc_pv = umma_idesc_bf16(BM, DV) | (1u << 16);
        const unsigned qa = desc_low(smem_u32(q_s) + i * Q_TILE, 1024), ka = desc_low(smem_u32(k_s), 1024), va = desc_low(smem_u32(v_s), KV_RUN);
        const unsigned st = tmem + 2 * i * KT, o = tmem + ROWS + i * BM;
        const bool one = elect_one();
        bool ok = i >= row_tiles || mbar_wait_compact(&bars->q_full, 0);
        // The scores of key tile t.  Their columns held the weights of tile t - 2: the product that read them must be done
        // (products into different accumulators are not ordered by their issue).
        auto scores = [&](int t) {
            if (t >= tiles || i >= row_tiles) return true;
            const int slot = t % KS;
            if ((t >= 2 && !mbar_wait_compact(&bars->o_done[i], t & 1)) || !mbar_wait_compact(&bars->k_full[slot], (t / KS) & 1)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (one) {
                const unsigned kt = ka + slot * (K_BYTES >> 4), s = st + (t & 1) * KT;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)  // 32 bytes further along k per step, 4 steps to a run
                    mma_ss(s, qa + (((ks >> 2) * Q_RUN + (ks & 3) * 32) >> 4), kt + (((ks >> 2) * KV_RUN + (ks & 3) * 32) >> 4), idesc_qk, ks > 0);
                umma_commit(&bars->s_done[2 * i + (t & 1)]);
                umma_commit(&bars->k_empty[slot]);
            }
            __syncwarp();
            return true;
        };
        // O += P V of key tile t
        auto values = [&](int t) {
            const int slot = t % VS;
            if (!mbar_wait_compact(&bars->v_full[slot], (t / VS) & 1) || !mbar_wait_compact(&bars->p_ready[2 * i + (t & 1)], (t >> 1) & 1)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (one) {
                const unsigned p = st + (t & 1) * KT, vt = va + slot * (V_BYTES >> 4);
#pragma unroll
                for (int term = 0; term < TERMS; ++term)
#pragma unroll
                    for (int ks = 0; ks < KT / 16; ++ks)  // 16 keys: 8 columns of weights, 2,048 bytes of values
                        mma_ts(o, p + term * 32 + ks * 8, vt + ks * (2048 >> 4), idesc_pv, term > 0 || ks > 0 || t > 0);
                umma_commit(&bars->o_done[i]);
                umma_commit(&bars->v_empty[slot]);
            }
            __syncwarp();
            return true;
        };
        const int mine = i < row_tiles ? tiles : 0;
        ok = ok && scores(0) && scores(1);
        for (int t = 0; t < mine && ok; ++t) ok = values(t) && scores(t + 2);
        if (!ok) bars->failed = 1;
    } else if (warp >= SOFTMAX_WARPS + MMA_WARPS) {
        // ---- copies: eight threads to a row of 128 bytes.  A tile's keys and values are one warp's, and the warps take turns: the fence
        // that hands the copies to the tensor core waits for all that its warp has in flight, so only other warps' copies go on beside it (two
        // warps that shared a tile and fenced keys and values apart took 2,600 clocks a tile, whatever the key size). ----
        const int w = warp - SOFTMAX_WARPS - MMA_WARPS, chunk = lane & 7, r0 = lane >> 3;
        constexpr int PASSES = KT / 4;
        // row r0 + 4 p: the same place in every other group of four rows
        const unsigned to0 = (unsigned)(r0 * 128 + ((chunk ^ r0) << 4)), to1 = (unsigned)((r0 + 4) * 128 + ((chunk ^ (r0 + 4)) << 4));
        auto place = [&](int p) { return (unsigned)(p >> 1) * 1024 + (p & 1 ? to1 : to0); };
        auto landed = [&]() {
            asm volatile("cp.async.wait_all;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
        };
        const int* table = FLAT ? nullptr : in.tables + (size_t)seq * in.table_width;
        int before = 0;  // FLAT: rows of the requests before this one
        if (FLAT)
            for (int i = 0; i < seq; ++i) before += in.ctx_lens[i];
        bool ok = true;
        // the row of each of the warp's keys, two to a lane, looked up while the copies before are in flight; -1: nothing there (reads as zero)
        int row_of[2] = {-1, -1};
        auto look_up = [&](int t) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int pos = key_of(t) + lane + 32 * j;
                row_of[j] = -1;
                if ((pos >= lo_min || pos < in.keep_first) && pos <= last_pos) {
                    if (FLAT) {
                        row_of[j] = before + pos;
                    } else {
                        const int page = table[pos >> in.page_shift];
                        if (page < 0 || page >= in.total_pages) {
                            ie_report(err, page < 0 ? IE_ERR_TABLE : IE_ERR_PAGE, page, q0 + row0 / group);
                        } else {
                            row_of[j] = ((page * in.kv_heads + kvh) << in.page_shift) + (pos & ((1 << in.page_shift) - 1));
                        }
                    }
                }
            }
        };
        if (w < tiles) look_up(w);
        for (int t = w; t < tiles; t += COPY_WARPS) {
            const int ks = t % KS, vs = t % VS;
            // (with three slots a warp meets a slot every other time it is filled; the time between is over, since the warp has waited for
            // a later tile's)
            if ((t >= KS && !mbar_wait_compact(&bars->k_empty[ks], (t / KS - 1) & 1)) ||
                (t >= VS && !mbar_wait_compact(&bars->v_empty[vs], (t / VS - 1) & 1))) { ok = false; break; }
            const unsigned kd = smem_u32(k_s) + ks * K_BYTES, vd = smem_u32(v_s) + vs * V_BYTES;
#pragma unroll 4
            for (int p = 0; p < PASSES; ++p) {
                const int row = __shfl_sync(0xffffffffu, p < PASSES / 2 ? row_of[0] : row_of[1], (r0 + 4 * p) & 31);
                const size_t at = (size_t)max(row, 0);
                const int bytes = row >= 0 ? 16 : 0;
                const bf16* k = in.k + (FLAT ? at * in.kv_ld + kvh * (D - 64) : at * D) + chunk * 8;
                const bf16* v = in.v + (FLAT ? at * in.kv_ld + kvh * DV : at * DV) + chunk * 8;
                const unsigned to = place(p);
#pragma unroll
                for (int h = 0; h < KH; ++h) {
                    if (FLAT && h == KH - 1) {
                        const bool rotated = row >= 0 && chunk * 8 < in.rot;
                        cp16(kd + to + h * KV_RUN, rotated ? in.k_rot + at * in.k_rot_ld + chunk * 8 : in.k, rotated ? 16 : 0);
                    } else {
                        cp16(kd + to + h * KV_RUN, k + h * 64, bytes);
                    }
                }
#pragma unroll
                for (int h = 0; h < VH; ++h) cp16(vd + to + h * KV_RUN, v + h * 64, bytes);
            }
            if (t + COPY_WARPS < tiles) look_up(t + COPY_WARPS);
            landed();
            if (lane == 0) {
                mbar_arrive(&bars->k_full[ks]);
                mbar_arrive(&bars->v_full[vs]);
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok) bars->failed = 1;
    } else {
        // ---- softmax: thread = row = tensor-memory lane ----
        const int i = warp >> 2, r = i * BM + (tid & (BM - 1));
        {   // the queries first, eight threads to 128 bytes of a row (while the copying warps fetch the first keys)
            const int chunk = lane & 7;
#pragma unroll 4
            for (int p = warp * 8; p < warp * 8 + 8; ++p) {
                const int qr = p * 4 + (lane >> 3);
                const bool there = qr < rows_here;
                const int rr = row0 + (there ? qr : 0), token = rr / group, head = kvh * group + rr - token * group;
                const size_t unit = (size_t)(q0 + token) * in.heads + head;
                const unsigned dst = smem_u32(q_s) + (qr >> 7) * Q_TILE + (qr & (BM - 1)) * 128 + ((chunk ^ (qr & 7)) << 4);
#pragma unroll
                for (int h = 0; h < KH; ++h) {
                    if (FLAT && h == KH - 1) {
                        const bool rotated = there && chunk * 8 < in.rot;
                        cp16(dst + h * Q_RUN, rotated ? in.q_rot + unit * in.q_rot_ld + chunk * 8 : in.q, rotated ? 16 : 0);
                    } else {
                        cp16(dst + h * Q_RUN, in.q + unit * (FLAT ? D - 64 : D) + chunk * 8 + h * 64, there ? 16 : 0);
                    }
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->q_full);
        }
        const bool exists = r < rows_here;
        const int rr = row0 + (exists ? r : 0), token = rr / group, head = kvh * group + rr - token * group;
        const int pos = exists ? start + token : -1, lo = in.window > 0 ? max(pos - in.window + 1, 0) : 0;
        // the first and the last position of the row tile (rows that do not exist follow its last)
        const int pos_lo = start + min(row0 + i * BM, rows_total - 1) / group;
        const int pos_hi = start + min(row0 + i * BM + BM - 1, rows_total - 1) / group;
        const unsigned lane_addr = (unsigned)((warp & 3) * 32) << 16;
        const unsigned to = tmem + ROWS + i * BM + lane_addr;
        const float sl2 = in.scale * LOG2E_F;
        const float cap_in = CAP ? in.scale / in.softcap : 0.f, cap_out = CAP ? in.softcap * LOG2E_F : 0.f;
        // m: the maximum that the weights are taken against (in units of log2 e); the sink is a term of the sum without key and value
        float m = in.sinks != nullptr ? in.sinks[head] * LOG2E_F : -INFINITY, l = in.sinks != nullptr ? 1.f : 0.f;
        bool ok = true;
        const int mine = i < row_tiles ? tiles : 0;
        for (int t = 0; t < mine; ++t) {
            const int key0 = key_of(t);
            if (!mbar_wait_compact(&bars->s_done[2 * i + (t & 1)], (t >> 1) & 1)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned ts = tmem + (2 * i + (t & 1)) * KT + lane_addr;
            const bool inner = key0 + KT - 1 <= pos_lo && (in.window <= 0 || key0 >= pos_hi - in.window + 1 || key0 + KT <= in.keep_first);
            float s[KT];
            tmem_ld64(s, ts);
            if (!inner) {
#pragma unroll
                for (int j = 0; j < KT; ++j) {
                    const int kp = key0 + j;
                    s[j] = kp <= pos && (kp >= lo || kp < in.keep_first) ? s[j] : -INFINITY;
                }
            }
            float mx[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) mx[j] = s[j];
#pragma unroll
            for (int j = 8; j < 56; j += 16)
#pragma unroll
                for (int k = 0; k < 8; ++k) mx[k] = max3(mx[k], s[j + k], s[j + 8 + k]);
#pragma unroll
            for (int k = 0; k < 8; ++k) mx[k] = fmaxf(mx[k], s[56 + k]);
            const float top = fmaxf(max3(max3(mx[0], mx[1], mx[2]), max3(mx[3], mx[4], mx[5]), mx[6]), mx[7]);
            // (scores are compared before scale and cap, which keep their order)
            const float m_seen = top == -INFINITY ? m : fmaxf(m, CAP ? cap_out * tanh_fast(top * cap_in) : top * sl2);
            const bool grown = m_seen > m + RESCALE_LAG;  // (from -inf: yes)
            const float alpha = grown ? fast_exp2(m - m_seen) : 1.f;
            if (grown) {
                m = m_seen;
                l *= alpha;
            }
            if (t > 0 && __any_sync(0xffffffffu, grown)) {
                // (the product of the tile before may still be running; the ones before that are done, since this tile's scores are)
                if (!mbar_wait_compact(&bars->o_done[i], (t - 1) & 1)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int d = 0; d < DV; d += 32) {
                    float acc[32];
                    tmem_ld32(acc, to + d);
#pragma unroll
                    for (int k = 0; k < 32; ++k) acc[k] *= alpha;
                    tmem_st32(acc, to + d);
                }
            }
            const float m_safe = m == -INFINITY ? 0.f : m;
            const float2 scale2 = make_float2(sl2, sl2), minus_m = make_float2(-m_safe, -m_safe), minus_one = make_float2(-1.f, -1.f);
            float2 sums[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                unsigned hi[16], rest[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const float s0 = s[part * 32 + 2 * k], s1 = s[part * 32 + 2 * k + 1];
                    float2 x;
                    if constexpr (CAP) {
                        x = make_float2(cap_out * tanh_fast(s0 * cap_in) - m_safe, cap_out * tanh_fast(s1 * cap_in) - m_safe);
                        if (!inner) {
                            if (s0 == -INFINITY) x.x = -INFINITY;
                            if (s1 == -INFINITY) x.y = -INFINITY;
                        }
                    } else {
                        x = fma2(make_float2(s0, s1), scale2, minus_m);
                    }
                    const float2 p = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                    sums[k & 1] = add2(sums[k & 1], p);
                    hi[k] = pack2(p.x, p.y);
                    if constexpr (TERMS == 2) {
                        const float2 r = fma2(as_float2(hi[k]), minus_one, p);  // (exact)
                        rest[k] = pack2(r.x, r.y);
                    }
                }
                tmem_st16(hi, ts + part * 16);
                if constexpr (TERMS == 2) tmem_st16(rest, ts + 32 + part * 16);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&bars->p_ready[2 * i + (t & 1)]);
            const float2 both = add2(sums[0], sums[1]);
            l += both.x + both.y;
        }
        // (the last scores only say that the product three tiles back is done: each of the two still open is waited for, since a wait for the
        // last alone would take the one before it for its like of two phases ago)
        if (ok && mine > 1) ok = mbar_wait_compact(&bars->o_done[i], tiles & 1);
        if (ok && mine > 0) ok = mbar_wait_compact(&bars->o_done[i], (tiles - 1) & 1);
        if (SHARED) {
            // (both row tiles' products are done and every copy has landed: queries, keys and values make room for the output)
            asm volatile("bar.sync 1, %0;" ::"n"(ROWS) : "memory");
            const bool filled = ok && mine > 0;
            *reinterpret_cast<float2*>(smem + ROWS * DV * 4 + r * 8) = make_float2(filled ? m : -INFINITY, filled ? l : 0.f);
            if (filled) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int d = 0; d < DV && i < row_tiles; d += 32) {
                float acc[32];
                if (filled) {
                    tmem_ld32(acc, to + d);
                } else {
#pragma unroll
                    for (int k = 0; k < 32; ++k) acc[k] = 0.f;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    *reinterpret_cast<float4*>(smem + r * (DV * 4) + (((d / 4 + k) ^ (r & 7)) << 4)) =
                        make_float4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]);
            }
        } else if (ok && i < row_tiles) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float f = l > 0.f ? 1.0f / l : 0.f;
            const float* gate = in.gate == nullptr ? nullptr : in.gate + (size_t)(q0 + token) * in.gate_ld + (in.gate_elements ? head * DV : head);
            if (gate != nullptr && !in.gate_elements) f *= 1.0f / (1.0f + expf(-gate[0]));
            bf16* out = in.out + (size_t)(q0 + token) * in.out_ld + head * DV;
#pragma unroll 1
            for (int d = 0; d < DV; d += 32) {
                float acc[32];
                tmem_ld32(acc, to + d);
                if (!exists) continue;
                if (gate != nullptr && in.gate_elements) {
#pragma unroll
                    for (int k = 0; k < 32; ++k) acc[k] *= 1.0f / (1.0f + expf(-gate[d + k]));
                }
#pragma unroll
                for (int k = 0; k < 32; k += 8)
                    *reinterpret_cast<uint4*>(out + d + k) = make_uint4(pack2(acc[k] * f, acc[k + 1] * f), pack2(acc[k + 2] * f, acc[k + 3] * f),
                                                                       pack2(acc[k + 4] * f, acc[k + 5] * f), pack2(acc[k + 6] * f, acc[k + 7] * f));
            }
        }
        if (!ok) bars->failed = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (SHARED) {
        cluster_barrier();
        add_shares(smem_u32(smem), smem_u32(smem) + ROWS * DV * 4, share, shares, in.out + (size_t)q0 * in.out_ld + kvh * group * DV, in.out_ld,
                   row0, rows_here, group, tid);
        cluster_barrier();  // (the others read this block's memory)
    }
    if (warp == SOFTMAX_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    if (tid == 0 && bars->failed) ie_report(err, IE_ERR_TIMEOUT, blockIdx.x, blockIdx.y);
}
}  // namespace

#if PA_PROMPT
// Plain softmax attention of a step's portions of more than 16 rows (tokens x heads of a group); the output has the queries' form.  `blocks`:
// at least the blocks of 256 rows that these portions have; the key tiles of each are shared among `shares` blocks (8 at most), a cluster.
IE_API int ie_attention_prompt(const void* q, const void* k_cache, const void* v_cache, const int* tables, int table_width, const int* cu_q,
                               const int* ctx_lens, void* out, int num_seqs, int blocks, int heads, int kv_heads, int page_size,
                               int total_pages, float scale, int window, int shares, int* err, void* stream) {
    if (num_seqs <= 0 || blocks <= 0) return 0;
    if (kv_heads <= 0 || heads % kv_heads != 0 || page_size < 1 || (page_size & (page_size - 1)) || window < 0 || shares < 1 ||
        shares > MOST_SHARES || (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) ||
        (long long)total_pages * kv_heads * page_size > 0x7fffffffll)
        return (int)cudaErrorInvalidValue;
    int page_shift = 0;
    while ((1 << page_shift) < page_size) ++page_shift;
    const Inputs in{(const bf16*)q, (const bf16*)k_cache, (const bf16*)v_cache, tables, cu_q, ctx_lens, table_width, heads, kv_heads,
                    page_shift, total_pages, scale, window, 0, 0.f, nullptr, nullptr, 0, 0, (bf16*)out, heads * DV,
                    nullptr, nullptr, 0, 0, 0, 0, num_seqs};
    static IePerDevice allowed, allowed_shared;
    cudaError_t e = ie_allow_smem(allowed, attention_packed_kernel<false, false>, SMEM_BYTES);
    if (e == cudaSuccess) e = ie_allow_smem(allowed_shared, attention_packed_kernel<false, true>, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid((unsigned)(blocks * kv_heads), shares);
    if (shares > 1) return ie_launch_cluster(attention_packed_kernel<false, true>, grid, dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream, dim3(1, shares, 1), in, err);
    return ie_launch(attention_packed_kernel<false, false>, grid, dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream, in, err);
}

// How many clusters of so many blocks the device runs at one time; 0: unknown.
IE_API int ie_attention_prompt_clusters(int shares) {
    if (shares < 1 || shares > MOST_SHARES) return 0;
    static IePerDevice allowed;
    if (ie_allow_smem(allowed, attention_packed_kernel<false, true>, SMEM_BYTES) != cudaSuccess) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, shares);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = (unsigned)shares;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, attention_packed_kernel<false, true>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return clusters;
}
#else
static int launch_packed(const Inputs& in, int num_seqs, int max_q_len, int* err, void* stream) {
    const long long rows = (long long)max_q_len * (in.heads / in.kv_heads);
    const dim3 grid((unsigned)((rows + ROWS - 1) / ROWS * in.kv_heads), num_seqs);
    static IePerDevice allowed, allowed_cap;
    cudaError_t e = ie_allow_smem(allowed, attention_packed_kernel<false, false>, SMEM_BYTES);
    if (e == cudaSuccess && !FLAT) e = ie_allow_smem(allowed_cap, attention_packed_kernel<!FLAT, false>, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    if (!FLAT && in.softcap > 0.f) return ie_launch(attention_packed_kernel<!FLAT, false>, grid, dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream, in, err);
    return ie_launch(attention_packed_kernel<false, false>, grid, dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream, in, err);
}

#if !PA_FLAT
// q: [tokens, heads, PA_D]; the caches [pages, kv_heads, page_size, PA_D or PA_DV]; out: rows of bfloat16 `out_ld` entries apart, 16-byte
// aligned, out_ld a multiple of 8.
IE_API int ie_attention_packed(const void* q, const void* k_cache, const void* v_cache, const int* tables, int table_width, const int* cu_q,
                               const int* ctx_lens, void* out, int num_seqs, int max_q_len, int heads, int kv_heads, int page_size,
                               int total_pages, float scale, int window, const float* sinks, const float* out_gate, int gate_ld,
                               int gate_elements, float softcap, int keep_first, int out_ld, int* err, void* stream) {
    if (num_seqs <= 0 || max_q_len <= 0) return 0;
    if (kv_heads <= 0 || heads % kv_heads != 0 || page_size < 1 || (page_size & (page_size - 1)) || window < 0 || softcap < 0.f ||
        keep_first < 0 || (window == 0 && keep_first > 0) || out_ld < heads * DV || out_ld % 8 ||
        (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) & 15) ||
        (long long)total_pages * kv_heads * page_size > 0x7fffffffll)
        return (int)cudaErrorInvalidValue;
    int page_shift = 0;
    while ((1 << page_shift) < page_size) ++page_shift;
    const Inputs in{(const bf16*)q, (const bf16*)k_cache, (const bf16*)v_cache, tables, cu_q, ctx_lens, table_width, heads, kv_heads,
                    page_shift, total_pages, scale, window, keep_first, softcap, sinks, out_gate, gate_ld, gate_elements, (bf16*)out, out_ld,
                    nullptr, nullptr, 0, 0, 0, 0, 0};
    return launch_packed(in, num_seqs, max_q_len, err, stream);
}
#else
// Every head has keys and values of its own.  q: [tokens, heads, PA_D - 64]; q_rot: the first of a (token, head)'s `rot` rotated entries
// (a multiple of 8 up to 64), q_rot_ld apart; kv: rows of kv_ld entries, all heads' keys (PA_D - 64 each), then all heads' values
// (PA_DV each), a row per context position, request after request; k_rot: such a row's shared rotated entries, k_rot_ld apart; out:
// [tokens, heads * PA_DV].  Everything 16-byte aligned, the distances multiples of 8.
IE_API int ie_attention_flat(const void* q, const void* q_rot, int q_rot_ld, const void* kv, int kv_ld, const void* k_rot, int k_rot_ld, int rot,
                             const int* cu_q, const int* ctx_lens, void* out, int num_seqs, int max_q_len, int heads, float scale,
                             const float* sinks, const float* out_gate, int gate_ld, int* err, void* stream) {
    if (num_seqs <= 0 || max_q_len <= 0) return 0;
    if (heads <= 0 || rot < 0 || rot > 64 || rot % 8 || q_rot_ld % 8 || k_rot_ld % 8 || kv_ld % 8 || kv_ld < heads * (D - 64 + DV) ||
        (((uintptr_t)q | (uintptr_t)q_rot | (uintptr_t)kv | (uintptr_t)k_rot | (uintptr_t)out) & 15))
        return (int)cudaErrorInvalidValue;
    const bf16* k = (const bf16*)kv;
    const Inputs in{(const bf16*)q, k, k + (size_t)heads * (D - 64), nullptr, cu_q, ctx_lens, 0, heads, heads, 0, 0, scale, 0, 0, 0.f, sinks,
                    out_gate, gate_ld, 0, (bf16*)out, heads * DV, (const bf16*)q_rot, (const bf16*)k_rot, q_rot_ld, k_rot_ld, kv_ld, rot, 0};
    return launch_packed(in, num_seqs, max_q_len, err, stream);
}
#endif
#endif
