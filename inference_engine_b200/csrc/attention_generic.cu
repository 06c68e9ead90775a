// Paged attention for any mix of prompt portions and decoded tokens, any head size that is
// a multiple of 8 up to 256, any number of heads and groups, 32-bit or bfloat16 cache.
//
// One warp per (token, query head).  The query at absolute position p of its request sees
// the keys at positions lo .. p of the same request (lo = 0, or p - window + 1 with a
// window), found through the request's block table.  Keys are walked in tiles of 32 aligned
// to absolute position 0; scores, the running maximum, the running sum and the weighted sum
// of values are 32-bit, with the same order of operations whatever else is in the step: a
// position's result depends on its own request's data only.  This is the attention of the
// engine's 32-bit path, and the fallback of the bfloat16 path for head sizes its
// tensor-core kernels do not take.  Counterparts in the reference:
// engine/kernels/paged_attention.py:44-87 (decode rows) and the gather + SDPA path
// engine/model/layers.py:215-225 (prompt portions).
// A value row may be shorter than a key row and may live inside it: `hdv` entries at the start of
// rows `v_stride` apart (a mixer that caches one shared latent row per token passes the key cache
// as the value cache too, `v_stride` = the key row and `hdv` = the latent's size).
// `chunk` > 0: a query sees only the keys of its own chunk of that many positions (counted from the
// request's position 0).  `head_bias` != null: the weight of a visible key is sigmoid(score +
// head_bias[head]) and the weights are not normalised over the keys (no softmax).
// `sinks` != null (softmax only): the denominator holds one more term exp(sinks[head]) that has no
// key and no value; it is the state the running maximum and sum start from.  `out_gate` != null:
// the head's result is multiplied by sigmoid(out_gate[token * gate_ld + head]).
// `softcap` > 0: a score s (after the scale) becomes softcap * tanh(s / softcap).  `keep_first` > 0 (with
// a window): the keys at positions below `keep_first` stay visible to every later query of the request,
// beside its window; they keep their own positions.
// A bias by distance n = (query's position - key's position), added to the score after the scale:
// -log_r1[head] * ln(1 + log_r2[head] * n), and/or a table, bias_table[head * bias_len + min(n, bias_len -
// 1)].  Rows of the output lie `out_ld` entries apart.  `gate_elements` 1: `out_gate` holds a number per head and value entry ([token * gate_ld + head *
// hdv + d]) instead of one per head.
#include "common.cuh"
#include <math.h>

namespace {
constexpr int WARPS = 4;
constexpr int MAX_ACC = 16;  // value rows of up to 512 entries

template <typename T>
__device__ __forceinline__ float dot_row_any(const float* __restrict__ q, const T* __restrict__ k, int hd) {
    float s = 0.f;  // (rows that are not a multiple of 16 bytes: one entry at a time)
    for (int d = 0; d < hd; ++d) s = fmaf(q[d], ie_load(k + d), s);
    return s;
}
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const float* __restrict__ k, int hd) {
    float s = 0.f;
    for (int d = 0; d < hd; d += 4) {
        float4 kv = *reinterpret_cast<const float4*>(k + d);
        s = fmaf(q[d], kv.x, s); s = fmaf(q[d + 1], kv.y, s);
        s = fmaf(q[d + 2], kv.z, s); s = fmaf(q[d + 3], kv.w, s);
    }
    return s;
}
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const __nv_bfloat16* __restrict__ k, int hd) {
    float s = 0.f;
    for (int d = 0; d < hd; d += 8) {
        uint4 raw = *reinterpret_cast<const uint4*>(k + d);
        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 f = __bfloat1622float2(h2[i]);
            s = fmaf(q[d + 2 * i], f.x, s);
            s = fmaf(q[d + 2 * i + 1], f.y, s);
        }
    }
    return s;
}

// One query row by one warp, `qs`: hd floats of the warp's own.
template <typename T>
__device__ __forceinline__ void
paged_attention_row(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                    const int* __restrict__ block_tables, int table_width, int token, int head, int seq, int pos, int lane,
                    float* qs, T* __restrict__ out,
                    int nh, int nkv, int hd, int hdv, int v_stride, int page_size, int total_pages,
                    float scale, int window, int chunk, const float* __restrict__ head_bias,
                    const float* __restrict__ sinks, const float* __restrict__ out_gate, int gate_ld,
                    float softcap, int keep_first, int gate_elements, const float* __restrict__ log_r1,
                    const float* __restrict__ log_r2, const float* __restrict__ bias_table, int bias_len,
                    int out_ld, int* err) {
    int kvh = head / (nh / nkv);
    const int* table = block_tables + (size_t)seq * table_width;
    const T* qrow = q + ((size_t)token * nh + head) * hd;
    for (int d = lane; d < hd; d += 32) qs[d] = ie_load(qrow + d);
    __syncwarp();

    int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    if (chunk > 0) lo = max(lo, (pos / chunk) * chunk);  // chunks are counted from the request's position 0
    const int kept = min(keep_first, lo);  // keys below `kept` are seen beside the window's
    const float inv_cap = softcap > 0.f ? 1.0f / softcap : 0.f;
    const bool gated = head_bias != nullptr;  // sigmoid(score + bias) per key, not normalised over keys
    float hb = gated ? head_bias[head] : 0.f;
    float m = -INFINITY, l = 0.f;
    if (!gated && sinks != nullptr) { m = sinks[head]; l = 1.0f; }
    float acc[MAX_ACC];
#pragma unroll
    for (int i = 0; i < MAX_ACC; ++i) acc[i] = 0.f;
    int nacc = (hdv + 31) / 32;

    for (int t0 = kept > 0 ? 0 : (lo / 32) * 32; t0 <= pos; t0 += 32) {
        if (t0 >= kept && t0 + 31 < lo) {  // between the kept keys and the window: nothing to see
            t0 = (lo / 32) * 32 - 32;
            continue;
        }
        int kpos = t0 + lane;
        bool valid = (kpos >= lo || kpos < kept) && kpos <= pos;
        long long row = -1;
        float s = -INFINITY;
        if (valid) {
            int page = table[kpos / page_size];
            if (page < 0 || page >= total_pages) {
                ie_report(err, page < 0 ? IE_ERR_TABLE : IE_ERR_PAGE, page, token);
                valid = false;
            } else {
                row = ((long long)page * nkv + kvh) * page_size + (kpos % page_size);
                s = (hd % 8 == 0 ? dot_row(qs, k_cache + row * hd, hd) : dot_row_any(qs, k_cache + row * hd, hd)) * scale;
                if (softcap > 0.f) s = softcap * tanhf(s * inv_cap);
                if (log_r1 != nullptr) s -= log_r1[head] * log1pf(log_r2[head] * (float)(pos - kpos));
                if (bias_table != nullptr) s += bias_table[(size_t)head * bias_len + min(pos - kpos, bias_len - 1)];
            }
        }
        float m_new = m, p;
        if (gated) {
            p = valid ? 1.0f / (1.0f + expf(-(s + hb))) : 0.f;
        } else {
            m_new = fmaxf(m, warp_max(s));
            p = valid ? expf(s - m_new) : 0.f;
            float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
            l = l * alpha + warp_sum(p);
#pragma unroll
            for (int i = 0; i < MAX_ACC; ++i) acc[i] *= alpha;
        }
        int count = min(32, pos - t0 + 1);
        for (int j = 0; j < count; ++j) {
            float pj = __shfl_sync(0xffffffffu, p, j);
            long long rj = __shfl_sync(0xffffffffu, row, j);
            if (rj < 0) continue;  // uniform across the warp
            const T* vrow = v_cache + rj * v_stride;
#pragma unroll
            for (int i = 0; i < MAX_ACC; ++i) {
                int d = lane + 32 * i;
                if (i < nacc && d < hdv) acc[i] = fmaf(pj, ie_load(vrow + d), acc[i]);
            }
        }
        m = m_new;
    }
    T* orow = out + (size_t)token * out_ld + (size_t)head * hdv;
    float inv = gated ? 1.0f : (l > 0.f ? 1.0f / l : 0.f);
    if (out_gate != nullptr && !gate_elements) inv *= 1.0f / (1.0f + expf(-out_gate[(size_t)token * gate_ld + head]));
#pragma unroll
    for (int i = 0; i < MAX_ACC; ++i) {
        int d = lane + 32 * i;
        if (i < nacc && d < hdv) {
            float f = inv;
            if (out_gate != nullptr && gate_elements)
                f *= 1.0f / (1.0f + expf(-out_gate[(size_t)token * gate_ld + (size_t)head * hdv + d]));
            ie_store(orow + d, acc[i] * f);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(WARPS * 32)
paged_attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_cache,
                               const T* __restrict__ v_cache, const int* __restrict__ block_tables,
                               int table_width, const int* __restrict__ seq_of_token,
                               const int* __restrict__ positions, T* __restrict__ out,
                               int nh, int nkv, int hd, int hdv, int v_stride, int page_size, int total_pages,
                               float scale, int window, int chunk, const float* __restrict__ head_bias,
                               const float* __restrict__ sinks, const float* __restrict__ out_gate, int gate_ld,
                               float softcap, int keep_first, int gate_elements, const float* __restrict__ log_r1,
                               const float* __restrict__ log_r2, const float* __restrict__ bias_table, int bias_len,
                               int out_ld, int* err) {
    extern __shared__ float q_smem[];  // [WARPS][hd]
    ie_pdl_trigger();
    ie_pdl_wait();
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int head = blockIdx.x * WARPS + warp;
    int token = blockIdx.y;
    if (head >= nh) return;  // whole warp leaves together; no block-wide barrier below
    paged_attention_row(q, k_cache, v_cache, block_tables, table_width, token, head, seq_of_token[token], positions[token], lane,
                        q_smem + warp * hd, out, nh, nkv, hd, hdv, v_stride, page_size, total_pages, scale, window, chunk, head_bias,
                        sinks, out_gate, gate_ld, softcap, keep_first, gate_elements, log_r1, log_r2, bias_table, bias_len, out_ld, err);
}

// The same attention for prompt portions in 32-bit (plain softmax, all positions or a window): a block takes 32 (token, query head of the
// group) rows of one request and key/value head and brings a tile of 32 keys once for all of them, where the kernel above reads a key
// row per warp and lane (377 tokens of 16 heads of 64 on 4: 221 us, here 45 by itself; 38 since no exponential
// is behind a branch and the products' loops are unrolled; a portion of 16 tokens behind 2,000 172 and 126).  Every number is the same chain of operations as there: a
// score one multiply-add after the other over the row, maxima and sums over a tile's 32 keys by the same exchanges (a warp
// takes a row, a lane a key), the output's multiply-adds key by key; tiles a row does not see leave it as it is (its maximum stays, a factor
// of 1, weights of 0).  So results are equal bit for bit, and a portion may be cut anywhere between the two kernels; where a value that some
// row does not see is infinite or not a number, or a page is not there, the block's rows go that kernel's way.  (Masks in the walk
// over the tiles: 2 to 10 % more time.)
constexpr int T_ROWS = 32, T_KEYS = 32, T_THREADS = 128;

// A block's rows by that kernel's own code, a warp a row.
template <int HD>
__device__ __noinline__ void
rows_one_by_one(const float* q, const float* k_cache, const float* v_cache, const int* block_tables, int table_width, int q0, int row0,
                int rows_here, int start, int seq, int kvh, float* q_smem, float* out, int nh, int nkv, int page_size, int total_pages,
                float scale, int window, int* err) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = nh / nkv;
    for (int rr = row0 + warp; rr < row0 + rows_here; rr += T_THREADS / 32) {
        const int token = rr / group, head = kvh * group + rr - token * group;
        paged_attention_row<float>(q, k_cache, v_cache, block_tables, table_width, q0 + token, head, seq, start + token, lane,
                                   q_smem + warp * HD, out, nh, nkv, HD, HD, HD, page_size, total_pages, scale, window, 0, nullptr, nullptr,
                                   nullptr, 0, 0.f, 0, 0, nullptr, nullptr, nullptr, 0, nh * HD, err);
        __syncwarp();
    }
}

// (Two blocks an SM at least, which leaves the compiler its registers: with the 86 of its own choice the loops are not interleaved.  256 threads
// a block took as long for few blocks and longer for many: what a tile costs is the chain through it.)
template <int HD>
__global__ void __launch_bounds__(T_THREADS, 2)
paged_attention_f32_tile_kernel(const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                                const int* __restrict__ block_tables, int table_width, const int* __restrict__ cu_q,
                                const int* __restrict__ ctx_lens, float* __restrict__ out, int nh, int nkv, int page_size, int total_pages,
                                float scale, int window, int* err) {
    constexpr int LD = HD + 4, LP = T_KEYS + 4;
    extern __shared__ __align__(16) float tile_smem[];
    float* qs = tile_smem;             // [32][LD]
    float* ks = qs + T_ROWS * LD;      // two of [32][LD]
    float* vs = ks + 2 * T_KEYS * LD;  // two of [32][HD]
    float* ps = vs + 2 * T_KEYS * HD;  // [32][LP]: scores, then weights
    float* alpha_s = ps + T_ROWS * LP; // [32]
    int* missing_s = reinterpret_cast<int*>(alpha_s + T_ROWS);  // a key that some row sees has no page
    ie_pdl_trigger();
    ie_pdl_wait();
    const int seq = blockIdx.z, kvh = blockIdx.y, group = nh / nkv, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q0 = cu_q[seq], q_len = cu_q[seq + 1] - q0, row0 = (gridDim.x - 1 - blockIdx.x) * T_ROWS, rows_total = q_len * group;
    if (row0 >= rows_total) return;
    const int start = ctx_lens[seq] - q_len, rows_here = min(T_ROWS, rows_total - row0);
    const int first_pos = start + row0 / group, last_pos = start + (row0 + rows_here - 1) / group;
    const int lo_min = window > 0 ? max(first_pos - window + 1, 0) : 0;
    const int* table = block_tables + (size_t)seq * table_width;
    if (tid == 0) *missing_s = 0;
    __syncthreads();
    auto fetch = [&](int t0, int b) {  // four threads a key
        const int key = tid >> 2, pos = t0 + key;
        int row = -1;
        if (pos >= lo_min && pos <= last_pos) {
            const int page = table[pos / page_size];
            if (page < 0 || page >= total_pages) {
                if ((tid & 3) == 0) ie_report(err, page < 0 ? IE_ERR_TABLE : IE_ERR_PAGE, page, q0 + row0 / group);
                *missing_s = 1;
            } else {
                row = (page * nkv + kvh) * page_size + pos % page_size;
            }
        }
        const float* kr = k_cache + (size_t)max(row, 0) * HD;
        const float* vr = v_cache + (size_t)max(row, 0) * HD;
#pragma unroll
        for (int c = (tid & 3) * 4; c < HD; c += 16) {
            const int bytes = row >= 0 ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(ks + (b * T_KEYS + key) * LD + c)), "l"(kr + c), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(vs + (b * T_KEYS + key) * HD + c)), "l"(vr + c), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int t_first = lo_min / T_KEYS * T_KEYS;
    fetch(t_first, 0);
    for (int i = tid; i < T_ROWS * HD / 4; i += T_THREADS) {
        const int r = i / (HD / 4), c = (i % (HD / 4)) * 4, rr = row0 + r, token = rr / group;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows_here) v = *reinterpret_cast<const float4*>(q + ((size_t)(q0 + token) * nh + kvh * group + rr - token * group) * HD + c);
        *reinterpret_cast<float4*>(qs + r * LD + c) = v;
    }
    // scores: 4 rows (8 apart) x 2 keys (16 apart) a thread; softmax: a warp every fourth row; output: 32 * HD / 128 numbers a thread
    const int sr = tid >> 4, sk = tid & 15;
    constexpr int DL = HD / 4, RG = T_THREADS / DL, OR = T_ROWS / RG;  // lanes across a row, rows at once, rows of a thread
    const int od = (tid % DL) * 4, orow = tid / DL;
    float m[T_ROWS / 4], l[T_ROWS / 4];
    int pos[T_ROWS / 4];
#pragma unroll
    for (int i = 0; i < T_ROWS / 4; ++i) { m[i] = -INFINITY; l[i] = 0.f; pos[i] = start + (row0 + warp + 4 * i) / group; }
    float acc[OR][4];
#pragma unroll
    for (int i = 0; i < OR; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    int b = 0;
    for (int t0 = t_first; t0 <= last_pos; t0 += T_KEYS, b ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the tile has landed, and everyone is done with the other one and with the weights
        if (t0 + T_KEYS <= last_pos) fetch(t0 + T_KEYS, b ^ 1);
        {
            const float* kt = ks + b * T_KEYS * LD;
            float s[4][2] = {};
#pragma unroll 16
            for (int d = 0; d < HD; d += 4) {
                float4 x[4], y[2];
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(qs + (sr + 8 * i) * LD + d);
#pragma unroll
                for (int j = 0; j < 2; ++j) y[j] = *reinterpret_cast<const float4*>(kt + (sk + 16 * j) * LD + d);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        s[i][j] = fmaf(x[i].x, y[j].x, s[i][j]); s[i][j] = fmaf(x[i].y, y[j].y, s[i][j]);
                        s[i][j] = fmaf(x[i].z, y[j].z, s[i][j]); s[i][j] = fmaf(x[i].w, y[j].w, s[i][j]);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) ps[(sr + 8 * i) * LP + sk + 16 * j] = s[i][j] * scale;
        }
        __syncthreads();
        {
            // (all rows' exchanges side by side; what rows beyond the block's give is not used)
            const int kpos = t0 + lane;
            float p[T_ROWS / 4], m_new[T_ROWS / 4], sum[T_ROWS / 4];
            bool valid[T_ROWS / 4];
#pragma unroll
            for (int i = 0; i < T_ROWS / 4; ++i) {
                valid[i] = kpos <= pos[i] && kpos >= (window > 0 ? max(pos[i] - window + 1, 0) : 0);
                p[i] = valid[i] ? ps[(warp + 4 * i) * LP + lane] : -INFINITY;
                m_new[i] = p[i];
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int i = 0; i < T_ROWS / 4; ++i) m_new[i] = fmaxf(m_new[i], __shfl_xor_sync(0xffffffffu, m_new[i], off));
#pragma unroll
            for (int i = 0; i < T_ROWS / 4; ++i) {
                m_new[i] = fmaxf(m[i], m_new[i]);
                p[i] = expf(valid[i] ? p[i] - m_new[i] : -INFINITY);  // (exactly 0, without a branch)
                sum[i] = p[i];
                ps[(warp + 4 * i) * LP + lane] = p[i];
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int i = 0; i < T_ROWS / 4; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], off);
#pragma unroll
            for (int i = 0; i < T_ROWS / 4; ++i) {
                const float alpha = expf(m[i] == -INFINITY ? m[i] : m[i] - m_new[i]);
                l[i] = fmaf(l[i], alpha, sum[i]);
                m[i] = m_new[i];
                if (lane == 0) alpha_s[warp + 4 * i] = alpha;
            }
        }
        __syncthreads();
        const float* vt = vs + b * T_KEYS * HD + od;
#pragma unroll
        for (int i = 0; i < OR; ++i) {
            const float a = alpha_s[orow + RG * i];
            acc[i][0] *= a; acc[i][1] *= a; acc[i][2] *= a; acc[i][3] *= a;
        }
#pragma unroll
        for (int j = 0; j < T_KEYS; j += 4) {
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = *reinterpret_cast<const float4*>(vt + (j + k) * HD);
#pragma unroll
            for (int i = 0; i < OR; ++i) {
                const float4 p = *reinterpret_cast<const float4*>(ps + (orow + RG * i) * LP + j);
                const float pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    acc[i][0] = fmaf(pv[k], v[k].x, acc[i][0]); acc[i][1] = fmaf(pv[k], v[k].y, acc[i][1]);
                    acc[i][2] = fmaf(pv[k], v[k].z, acc[i][2]); acc[i][3] = fmaf(pv[k], v[k].w, acc[i][3]);
                }
            }
        }
    }
    __syncthreads();  // (the last tile's factors have been read)
#pragma unroll
    for (int i = 0; i < T_ROWS / 4; ++i) {
        const int r = warp + 4 * i;
        if (lane == 0 && r < rows_here) alpha_s[r] = l[i] > 0.f ? 1.0f / l[i] : 0.f;
    }
    __syncthreads();
    // A hidden value has a weight of 0 and changes nothing, unless it is infinite or not a number: then an output is not a number.
    float z = 0.f;
#pragma unroll
    for (int i = 0; i < OR; ++i) {
        const int r = orow + RG * i, rr = row0 + r, token = rr / group;
        if (r >= rows_here) continue;
        const float f = alpha_s[r];
        const float4 o = make_float4(acc[i][0] * f, acc[i][1] * f, acc[i][2] * f, acc[i][3] * f);
        z += (o.x + o.y + o.z + o.w) * 0.f;
        *reinterpret_cast<float4*>(out + ((size_t)(q0 + token) * nh + kvh * group + rr - token * group) * HD + od) = o;
    }
    if (__syncthreads_or(z != 0.f || *missing_s))
        rows_one_by_one<HD>(q, k_cache, v_cache, block_tables, table_width, q0, row0, rows_here, start, seq, kvh, tile_smem, out, nh, nkv,
                            page_size, total_pages, scale, window, err);
}

template <int HD>
int launch_f32_tile(const float* q, const float* k, const float* v, const int* tables, int width, const int* cu_q, const int* ctx_lens,
                    float* out, int num_seqs, int max_q_len, int nh, int nkv, int page_size, int total_pages, float scale, int window,
                    int* err, cudaStream_t s) {
    constexpr size_t smem = (size_t)(T_ROWS * (HD + 4) + 2 * T_KEYS * (HD + 4) + 2 * T_KEYS * HD + T_ROWS * (T_KEYS + 4) + T_ROWS + 1) * sizeof(float);
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, paged_attention_f32_tile_kernel<HD>, smem);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid((unsigned)(((long long)max_q_len * (nh / nkv) + T_ROWS - 1) / T_ROWS), nkv, num_seqs);
    return ie_launch(paged_attention_f32_tile_kernel<HD>, grid, dim3(T_THREADS), smem, s, q, k, v, tables, width, cu_q, ctx_lens, out, nh,
                     nkv, page_size, total_pages, scale, window, err);
}
}  // namespace

IE_API int ie_paged_attention_generic(const void* q, const void* k_cache, const void* v_cache,
                                      int dtype, const int* block_tables, int table_width,
                                      const int* seq_of_token, const int* positions, void* out,
                                      int num_tokens, int nh, int nkv, int hd, int hdv, int v_stride,
                                      int page_size, int total_pages, float scale, int window, int chunk,
                                      const float* head_bias, const float* sinks, const float* out_gate,
                                      int gate_ld, float softcap, int keep_first, int gate_elements,
                                      const float* log_r1, const float* log_r2, const float* bias_table,
                                      int bias_len, int out_ld, int* err, void* stream) {
    if (num_tokens <= 0) return 0;
    if (hd < 1 || hdv < 1 || hdv > 32 * MAX_ACC || nkv <= 0 || nh % nkv != 0 || out_ld < nh * hdv) return (int)cudaErrorInvalidValue;
    if (keep_first < 0 || softcap < 0.f || (keep_first > 0 && chunk > 0)) return (int)cudaErrorInvalidValue;
    if ((log_r1 == nullptr) != (log_r2 == nullptr) || (bias_table != nullptr && bias_len < 1))
        return (int)cudaErrorInvalidValue;
    dim3 grid((nh + WARPS - 1) / WARPS, num_tokens);
    size_t smem = (size_t)WARPS * hd * sizeof(float);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == IE_BF16)
        paged_attention_generic_kernel<<<grid, WARPS * 32, smem, s>>>(
            (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache,
            block_tables, table_width, seq_of_token, positions, (__nv_bfloat16*)out,
            nh, nkv, hd, hdv, v_stride, page_size, total_pages, scale, window, chunk, head_bias, sinks, out_gate, gate_ld, softcap, keep_first,
            gate_elements, log_r1, log_r2, bias_table, bias_len, out_ld, err);
    else
        paged_attention_generic_kernel<<<grid, WARPS * 32, smem, s>>>(
            (const float*)q, (const float*)k_cache, (const float*)v_cache,
            block_tables, table_width, seq_of_token, positions, (float*)out,
            nh, nkv, hd, hdv, v_stride, page_size, total_pages, scale, window, chunk, head_bias, sinks, out_gate, gate_ld, softcap, keep_first,
            gate_elements, log_r1, log_r2, bias_table, bias_len, out_ld, err);
    return IE_LAUNCH_CHECK();
}

// 32-bit prompt portions with rows of 32, 64 or 128 entries; everything 16-byte aligned.
IE_API int ie_paged_attention_f32_tiles(const float* q, const float* k_cache, const float* v_cache, const int* tables, int table_width,
                                        const int* cu_q, const int* ctx_lens, float* out, int num_seqs, int max_q_len, int nh, int nkv, int hd,
                                        int page_size, int total_pages, float scale, int window, int* err, void* stream) {
    if (num_seqs <= 0 || max_q_len <= 0) return 0;
    if (nkv <= 0 || nh % nkv || page_size < 1 || window < 0 || (long long)total_pages * nkv * page_size > 0x7fffffffll) return (int)cudaErrorInvalidValue;
#define IE_F32_TILE(HD)                                                                                                              \
    if (hd == HD)                                                                                                                    \
    return launch_f32_tile<HD>(q, k_cache, v_cache, tables, table_width, cu_q, ctx_lens, out, num_seqs, max_q_len, nh, nkv, page_size, \
                               total_pages, scale, window, err, (cudaStream_t)stream)
    IE_F32_TILE(32);
    IE_F32_TILE(64);
    IE_F32_TILE(128);
#undef IE_F32_TILE
    return (int)cudaErrorInvalidValue;
}
