// Softmax attention of prompt portions on the fifth-generation tensor cores, bfloat16, with what the engine's softmax mixers ask
// for: a sink, a sliding window beside kept first positions, capped scores, an output gate.  Built per (key size PA_D: 64, 128 or 192;
// value size PA_DV: 64 or 128).
//
// A block owns 256 rows of one request and one key/value head, a row being a (token, query head of the group) pair, so that a key tile
// is brought once for the whole group, and walks tiles of 128 keys.  Two row tiles of 128 take turns: while the softmax warps of one work, the
// tensor core serves the other.  Eleven warps (with a thirteenth a thread would have 128 registers instead of 168, and spill):
//   warps 0-3, 4-7: softmax of row tile 0 and 1, a thread per row (tensor-memory lane);
//   warp 8: tcgen05.mma.  Per key tile and row tile: O += P V of the tile before (P, in tensor memory, over the scores it was made
//     from), then S = Q K^T (both from shared memory).  The whole warp runs the loop and one elected lane issues, so that
//     descriptors stay in uniform registers;
//   warps 9, 10: gather keys and values from the request's pages by cp.async, swizzled by hand as the tensor core reads them.  (Pages of
//     16 tokens as TMA boxes are 2 KB each, and the copy engine spends some 300 clocks on any box: 32 of them per key tile would take three
//     times as long as the tile's products.)
// Tensor memory: scores of the row tiles in columns 0 and 128, their outputs in 256 and 384.  A row's weights replace its scores 64 keys at a
// time: 32 columns of weights rounded to bfloat16, two to a column, then 32 columns of what the rounding left (TERMS 2: a weight keeps 16 bits of
// mantissa; both go through the second product).  The maximum that weights are taken against follows a row's running maximum only when that
// has grown by more than 2^8; only then is the row's output rescaled.  A row's arithmetic depends on its own request alone.
//
// What bounds it: the special-function unit (128 x 256 exponentials a key tile: 2,048 clocks) beside the products (head size 128: 1,536 clocks).
// Sixteen query heads on four of 128, window 1,024, 2,048 tokens: the mma.sync kernel that serves the other sizes takes 148 us.
// Every wait is bounded; a block that waits too long records IE_ERR_TIMEOUT, frees its tensor memory and leaves.
#include "tma.cuh"
#include <math.h>

#ifndef PA_D
#define PA_D 128
#endif
#ifndef PA_DV
#define PA_DV 128
#endif

using namespace ie_tma;

namespace {
constexpr int D = PA_D, DV = PA_DV;
static_assert((D == 64 || D == 128 || D == 192) && (DV == 64 || DV == 128), "sizes");
constexpr int TERMS = 2;
constexpr int BM = 128, ROWS = 2 * BM, KT = 128;
constexpr int KH = D / 64, VH = DV / 64;         // runs of 64 entries: 128 bytes, one swizzle atom
constexpr int HALF = KT * 128;                   // such a run of a tile's 128 rows: 16 KB
constexpr int K_BYTES = KH * HALF, V_BYTES = VH * HALF, Q_BYTES = 2 * K_BYTES;
constexpr int KS = D == 64 ? 4 : 2, VS = DV == 64 ? 4 : D == 192 ? 1 : 2;  // tiles of keys and of values in shared memory
constexpr int SOFTMAX_WARPS = 8, COPY_WARPS = 2, THREADS = (SOFTMAX_WARPS + 1 + COPY_WARPS) * 32;
constexpr float RESCALE_LAG = 8.0f;              // in powers of two
constexpr float LOG2E_F = 1.4426950408889634f;

struct __align__(8) Bars {
    unsigned long long q_full, k_full[KS], k_empty[KS], v_full[VS], v_empty[VS], s_done[2], p_ready[2], o_done[2];
    unsigned tmem_base;
    int failed;
};
constexpr size_t SMEM_BYTES = (size_t)Q_BYTES + KS * K_BYTES + VS * V_BYTES + sizeof(Bars) + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
// B with its N entries contiguous (values: 64 entries to 128 bytes, runs of 64 `run` bytes apart, eight keys to 1,024 bytes).
__device__ __forceinline__ unsigned long long desc_mn(unsigned addr, unsigned run) {
    unsigned long long d = 0;
    d |= (unsigned long long)((addr >> 4) & 0x3FFF);
    d |= (unsigned long long)((run >> 4) & 0x3FFF) << 16;
    d |= (unsigned long long)64 << 32;
    d |= (unsigned long long)1 << 46;
    d |= (unsigned long long)2 << 61;
    return d;
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
};

// grid: (blocks of 256 rows of the longest portion, key/value heads, requests)
template <bool CAP>
__global__ void __launch_bounds__(THREADS, 1)
attention_packed_kernel(const Inputs in, int* err) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* q_s = smem;                      // [row tile][run][128 rows][128 bytes]
    unsigned char* k_s = q_s + Q_BYTES;             // [slot][run][128 keys][128 bytes]
    unsigned char* v_s = k_s + KS * K_BYTES;
    Bars* bars = reinterpret_cast<Bars*>(v_s + VS * V_BYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    ie_pdl_trigger();
    // (lengths and block tables are the step's inputs; queries, keys and values are the kernels' before)
    const int seq = blockIdx.z, kvh = blockIdx.y, group = in.heads / in.kv_heads;
    const int q0 = in.cu_q[seq], q_len = in.cu_q[seq + 1] - q0;
    const int row0 = (gridDim.x - 1 - blockIdx.x) * ROWS, rows_total = q_len * group;  // (the rows that see most start first)
    if (row0 >= rows_total) return;
    const int start = in.ctx_lens[seq] - q_len;  // position of the request's first token of this step
    const int rows_here = min(ROWS, rows_total - row0);
    const int first_pos = start + row0 / group, last_pos = start + (row0 + rows_here - 1) / group;
    const int lo_min = in.window > 0 ? max(first_pos - in.window + 1, 0) : 0;
    // the tiles the block walks, by a running number: those that hold kept keys and lie before the window's first, then the window's
    const int win_begin = lo_min / KT, win_end = last_pos / KT;
    const int kept_tiles = in.keep_first > 0 ? min((in.keep_first - 1) / KT + 1, win_begin) : 0;
    const int tiles = kept_tiles + win_end - win_begin + 1;
    auto key_of = [&](int t) { return (t < kept_tiles ? t : win_begin + t - kept_tiles) * KT; };

    if (tid == 0) {
        mbar_init(&bars->q_full, COPY_WARPS);
        for (int s = 0; s < KS; ++s) { mbar_init(&bars->k_full[s], COPY_WARPS); mbar_init(&bars->k_empty[s], 1); }
        for (int s = 0; s < VS; ++s) { mbar_init(&bars->v_full[s], COPY_WARPS); mbar_init(&bars->v_empty[s], 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->s_done[i], 1);
            mbar_init(&bars->p_ready[i], BM);
            mbar_init(&bars->o_done[i], 1);
        }
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
    const unsigned tmem = bars->tmem_base;
    ie_pdl_wait();

    if (warp == SOFTMAX_WARPS) {
        // ---- tensor core ----
        const unsigned idesc_qk = umma_idesc_bf16(BM, KT), idesc_pv = umma_idesc_bf16(BM, DV) | (1u << 16);
        const unsigned qa = smem_u32(q_s), ka = smem_u32(k_s), va = smem_u32(v_s);
        const bool one = elect_one();
        bool ok = mbar_wait_compact(&bars->q_full, 0);
        for (int t = 0; t <= tiles && ok; ++t) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (t > 0) {  // the tile before: its weights are written
                    const int slot = (t - 1) % VS;
                    ok = ok && (i > 0 || mbar_wait_compact(&bars->v_full[slot], ((t - 1) / VS) & 1)) &&
                         mbar_wait_compact(&bars->p_ready[i], (t - 1) & 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (one) {
                        const unsigned p = tmem + i * KT, o = tmem + ROWS + i * BM, vt = va + slot * V_BYTES;
#pragma unroll
                        for (int term = 0; term < TERMS; ++term)
#pragma unroll
                            for (int ks = 0; ks < KT / 16; ++ks)  // 16 keys: 8 columns of weights, 2,048 bytes of values
                                umma_ta(o, p + (ks >> 2) * 64 + term * 32 + (ks & 3) * 8, desc_mn(vt + ks * 2048, HALF), idesc_pv,
                                        t > 1 || term > 0 || ks > 0 ? 1u : 0u);
                        if (t == tiles) umma_commit(&bars->o_done[i]);
                        if (i == 1) umma_commit(&bars->v_empty[slot]);
                    }
                    __syncwarp();
                }
                if (t < tiles) {
                    const int slot = t % KS;
                    if (i == 0) ok = mbar_wait_compact(&bars->k_full[slot], (t / KS) & 1);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (one) {
                        const unsigned qt = qa + i * K_BYTES, kt = ka + slot * K_BYTES;
#pragma unroll
                        for (int ks = 0; ks < D / 16; ++ks)  // 32 bytes further along k per step, 4 steps to a run
                            umma_ss(tmem + i * KT, umma_desc_sw128(qt + (ks >> 2) * HALF + (ks & 3) * 32),
                                    umma_desc_sw128(kt + (ks >> 2) * HALF + (ks & 3) * 32), idesc_qk, ks > 0 ? 1u : 0u);
                        umma_commit(&bars->s_done[i]);
                        if (i == 1) umma_commit(&bars->k_empty[slot]);
                    }
                    __syncwarp();
                }
            }
        }
        if (!ok) bars->failed = 1;
    } else if (warp > SOFTMAX_WARPS) {
        // ---- copies: eight threads to a row of 128 bytes, eight rows at a time ----
        const int c = tid - (SOFTMAX_WARPS + 1) * 32, chunk = c & 7, r0 = c >> 3;
        const unsigned to = (unsigned)(r0 * 128 + ((chunk ^ (r0 & 7)) << 4));  // (r0 + 8 p: the same place in its group of eight rows)
        constexpr int AT_ONCE = COPY_WARPS * 4, PASSES = KT / AT_ONCE;
        static_assert(AT_ONCE == 8, "rows at a time");
        // what was asked for last and not announced yet
        unsigned long long* pending = nullptr;
        auto announce = [&](unsigned long long* bar) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        auto settle = [&](bool all) {  // the copies before the last group have landed, or all of them
            if (all) asm volatile("cp.async.wait_group 0;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            if (pending != nullptr) announce(pending);
            pending = nullptr;
        };
        auto asked = [&](unsigned long long* bar) {
            asm volatile("cp.async.commit_group;" ::: "memory");
            settle(false);
            pending = bar;
        };
        // a slot that is not free yet: whatever is on its way is announced before the wait, since the slot may depend on it
        auto slot_free = [&](unsigned long long* bar, int parity) {
            settle(true);
            return mbar_wait_compact(bar, parity);
        };
        {
            #pragma unroll 4
            for (int p = 0; p < ROWS / AT_ONCE; ++p) {
                const int r = r0 + AT_ONCE * p;
                const bool there = r < rows_here;
                const int rr = row0 + (there ? r : 0), token = rr / group, head = kvh * group + rr - token * group;
                const bf16* src = in.q + ((size_t)(q0 + token) * in.heads + head) * D + chunk * 8;
                const unsigned dst = smem_u32(q_s) + (r >> 7) * K_BYTES + (p & (PASSES - 1)) * 1024 + to;
#pragma unroll
                for (int h = 0; h < KH; ++h) cp16(dst + h * HALF, src + h * 64, there ? 16 : 0);
            }
            asked(&bars->q_full);
        }
        const int* table = in.tables + (size_t)seq * in.table_width;
        bool ok = true;
        for (int t = 0; t < tiles; ++t) {
            const int key0 = key_of(t);
            int row[PASSES];  // the cache's row of each of the thread's keys; -1: nothing there (reads as zero)
#pragma unroll
            for (int p = 0; p < PASSES; ++p) {
                const int pos = key0 + r0 + AT_ONCE * p;
                row[p] = -1;
                if ((pos >= lo_min || pos < in.keep_first) && pos <= last_pos) {
                    const int page = table[pos >> in.page_shift];
                    if (page < 0 || page >= in.total_pages) {
                        if (chunk == 0) ie_report(err, page < 0 ? IE_ERR_TABLE : IE_ERR_PAGE, page, q0 + row0 / group);
                    } else {
                        row[p] = ((page * in.kv_heads + kvh) << in.page_shift) + (pos & ((1 << in.page_shift) - 1));
                    }
                }
            }
            const int ks = t % KS, vs = t % VS;
            if (t >= KS && !slot_free(&bars->k_empty[ks], (t / KS - 1) & 1)) { ok = false; break; }
            unsigned dst = smem_u32(k_s) + ks * K_BYTES + to;
#pragma unroll
            for (int p = 0; p < PASSES; ++p) {
                const bf16* src = in.k + (size_t)max(row[p], 0) * D + chunk * 8;
#pragma unroll
                for (int h = 0; h < KH; ++h) cp16(dst + p * 1024 + h * HALF, src + h * 64, row[p] >= 0 ? 16 : 0);
            }
            asked(&bars->k_full[ks]);
            if (t >= VS && !slot_free(&bars->v_empty[vs], (t / VS - 1) & 1)) { ok = false; break; }
            dst = smem_u32(v_s) + vs * V_BYTES + to;
#pragma unroll
            for (int p = 0; p < PASSES; ++p) {
                const bf16* src = in.v + (size_t)max(row[p], 0) * DV + chunk * 8;
#pragma unroll
                for (int h = 0; h < VH; ++h) cp16(dst + p * 1024 + h * HALF, src + h * 64, row[p] >= 0 ? 16 : 0);
            }
            asked(&bars->v_full[vs]);
        }
        settle(true);
        if (!ok) bars->failed = 1;
    } else {
        // ---- softmax: thread = row = tensor-memory lane ----
        const int i = warp >> 2, r = i * BM + (tid & (BM - 1));
        const bool exists = r < rows_here;
        const int rr = row0 + (exists ? r : 0), token = rr / group, head = kvh * group + rr - token * group;
        const int pos = exists ? start + token : -1, lo = in.window > 0 ? max(pos - in.window + 1, 0) : 0;
        // the first and the last position of the row tile (rows that do not exist follow its last)
        const int pos_lo = start + min(row0 + i * BM, rows_total - 1) / group;
        const int pos_hi = start + min(row0 + i * BM + BM - 1, rows_total - 1) / group;
        const unsigned lane_addr = (unsigned)((warp & 3) * 32) << 16;
        const unsigned ts = tmem + i * KT + lane_addr, to = tmem + ROWS + i * BM + lane_addr;
        const float sl2 = in.scale * LOG2E_F;
        const float cap_in = CAP ? in.scale / in.softcap : 0.f, cap_out = CAP ? in.softcap * LOG2E_F : 0.f;
        // m: the maximum that the weights are taken against (in units of log2 e); the sink is a term of the sum without key and value
        float m = in.sinks != nullptr ? in.sinks[head] * LOG2E_F : -INFINITY, l = in.sinks != nullptr ? 1.f : 0.f;
        bool ok = true;
        for (int t = 0; t < tiles; ++t) {
            const int key0 = key_of(t);
            if (!mbar_wait_compact(&bars->s_done[i], t & 1)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool inner = key0 + KT - 1 <= pos_lo && (in.window <= 0 || key0 >= pos_hi - in.window + 1 || key0 + KT <= in.keep_first);
            float s[64];
            auto scores = [&](int half) {
                tmem_ld64(s, ts + half * 64);
                if (!inner) {
#pragma unroll
                    for (int j = 0; j < 64; ++j) {
                        const int kp = key0 + half * 64 + j;
                        s[j] = kp <= pos && (kp >= lo || kp < in.keep_first) ? s[j] : -INFINITY;
                    }
                }
            };
            auto maximum = [&](float before) {
                float mx[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) mx[j] = s[j];
#pragma unroll
                for (int j = 8; j < 56; j += 16)
#pragma unroll
                    for (int k = 0; k < 8; ++k) mx[k] = max3(mx[k], s[j + k], s[j + 8 + k]);
#pragma unroll
                for (int k = 0; k < 8; ++k) mx[k] = fmaxf(mx[k], s[56 + k]);
                return fmaxf(before, fmaxf(max3(max3(mx[0], mx[1], mx[2]), max3(mx[3], mx[4], mx[5]), mx[6]), mx[7]));
            };
            scores(0);
            float top = maximum(-INFINITY);
            scores(1);
            top = maximum(top);
            // (scores are compared before scale and cap, which keep their order)
            const float m_seen = top == -INFINITY ? m : fmaxf(m, CAP ? cap_out * tanh_fast(top * cap_in) : top * sl2);
            const bool grown = m_seen > m + RESCALE_LAG;  // (from -inf: yes)
            const float alpha = grown ? fast_exp2(m - m_seen) : 1.f;
            if (grown) {
                m = m_seen;
                l *= alpha;
            }
            if (t > 0 && __any_sync(0xffffffffu, grown)) {  // (the products before this tile's scores are done)
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
            const float2 scale2 = make_float2(sl2, sl2), minus_m = make_float2(-m_safe, -m_safe);
            float2 sums[2] = {{0.f, 0.f}, {0.f, 0.f}};
            auto weights = [&](int half) {
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
                        const float2 r = as_float2(hi[k]);
                        rest[k] = pack2(p.x - r.x, p.y - r.y);
                    }
                    tmem_st16(hi, ts + half * 64 + part * 16);
                    tmem_st16(rest, ts + half * 64 + 32 + part * 16);
                }
            };
            weights(1);
            scores(0);  // (the first half's scores once more: both halves at once would not fit the registers)
            weights(0);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            const float2 both = add2(sums[0], sums[1]);
            l += both.x + both.y;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&bars->p_ready[i]);
        }
        if (ok) ok = mbar_wait_compact(&bars->o_done[i], 0);
        if (ok) {
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
    if (warp == SOFTMAX_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    if (tid == 0 && bars->failed) ie_report(err, IE_ERR_TIMEOUT, blockIdx.x, blockIdx.y);
}
}  // namespace

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
                    page_shift, total_pages, scale, window, keep_first, softcap, sinks, out_gate, gate_ld, gate_elements, (bf16*)out, out_ld};
    const long long rows = (long long)max_q_len * (heads / kv_heads);
    const dim3 grid((unsigned)((rows + ROWS - 1) / ROWS), kv_heads, num_seqs);
    static IePerDevice allowed, allowed_cap;
    cudaError_t e = ie_allow_smem(allowed, attention_packed_kernel<false>, SMEM_BYTES);
    if (e == cudaSuccess) e = ie_allow_smem(allowed_cap, attention_packed_kernel<true>, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    if (softcap > 0.f) return ie_launch(attention_packed_kernel<true>, grid, dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream, in, err);
    return ie_launch(attention_packed_kernel<false>, grid, dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream, in, err);
}
