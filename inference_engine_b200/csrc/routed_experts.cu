// Kernels of the routed feed-forward (many small gated experts, a few per token).
//
//  * route_topk: per token the router's logits (32-bit; plus a bias per expert if the router has
//    one), their softmax over all experts, the
//    groups' best scores, the kept groups, the `top` best allowed experts (ties: the lower index)
//    and their scores divided by their sum (+ 1e-20), times `weight_scale`.  With `sigmoid_scores` an
//    expert's score is the sigmoid of its logit instead; a `correction` per expert is then added for
//    the choice alone (groups and experts are chosen by score + correction, the weights are the plain
//    scores), a group is ranked by its best `group_top` (1 or 2) corrected scores added up, and the
//    experts of groups that are not kept cannot be chosen whatever their sign.
//  * routed_align: the step's (token, choice) pairs sorted by expert into tiles of TILE_M rows:
//    every expert's run of pairs is padded to whole tiles (padding rows are -1), and a list says
//    which expert each tile belongs to.  One block; nothing goes to the host.
//  * routed_gate_up: per tile and 64 columns: gate and up products of the tile's tokens with the
//    tile's expert, then  g = min(gate, limit), u = clamp(up, -limit, limit),
//    y = g * sigmoid(alpha * g) * (u + up_offset), written per pair.
//  * routed_down: per tile and 64 columns: y times the expert's down matrix, times the pair's
//    routing weight, written to out[choice][token][:]; the consumer adds the `top` slices in order.
// bfloat16 products run on mma.sync.m16n8k16 with 32-bit sums, 32-bit products on fused
// multiply-adds; a row's sums run over k in a fixed order, whatever else is in the tile.
#include "common.cuh"
#include <limits.h>
#include <math.h>

namespace {

// The lane's best of `count` scores (larger first, then the lower index), over the warp: every lane gets the index, -1 if no score
// is above `floor` (one that is no number is above nothing).
__device__ __forceinline__ int warp_best(const float* score, int count, float floor, int lane) {
    float bv = floor;
    int best = INT_MAX;
    for (int e = lane; e < count; e += 32)
        if (score[e] > bv) { bv = score[e]; best = e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best, o);
        if (ov > bv || (ov == bv && oi < best)) { bv = ov; best = oi; }
    }
    return best == INT_MAX ? -1 : best;
}

// A warp chooses token n's experts from their logits (score[experts]; gbest[groups] and choice[experts] are its scratch).
__device__ __forceinline__ void choose_experts(int n, float* score, float* gbest, float* choice, int lane, int experts, int top, int groups,
                                               int keep, int sigmoid_scores, const float* __restrict__ correction, int group_top,
                                               float weight_scale, int* __restrict__ ids, float* __restrict__ weights) {
    const int per = experts / groups;
    float total = 0.f;
    if (sigmoid_scores) {
        for (int e = lane; e < experts; e += 32) {
            float sg = 1.0f / (1.0f + expf(-score[e]));
            score[e] = sg;
            choice[e] = correction != nullptr ? sg + correction[e] : sg;
        }
        __syncwarp();
        if (keep < groups) {
            for (int g = lane; g < groups; g += 32) {  // the group's best corrected scores, one or two of them
                float b1 = -INFINITY, b2 = -INFINITY;
                for (int e = g * per; e < (g + 1) * per; ++e) {
                    float c = choice[e];
                    if (c > b1) { b2 = b1; b1 = c; }
                    else if (c > b2) b2 = c;
                }
                gbest[g] = (group_top >= 2 && per >= 2) ? b1 + b2 : b1;
            }
            __syncwarp();
            // The kept groups are marked by +inf.  (A group without any score to compare counts as the lowest, not as none: when nothing
            // better is left it is kept, the one with the lowest index first.)
            for (int round = 0; round < keep; ++round) {
                int best = -1;
                if (lane == 0) {
                    float bv = -INFINITY;
                    for (int g = 0; g < groups; ++g)
                        if (gbest[g] != INFINITY && (best < 0 || gbest[g] > bv)) { bv = gbest[g]; best = g; }
                    if (best >= 0) gbest[best] = INFINITY;
                }
                if (__shfl_sync(0xffffffffu, best, 0) < 0) break;
            }
            __syncwarp();
            for (int e = lane; e < experts; e += 32)
                if (gbest[e / per] != INFINITY) choice[e] = -INFINITY;
            __syncwarp();
        }
        for (int j = 0; j < top; ++j) {
            const int best = warp_best(choice, experts, -INFINITY, lane);
            const float wj = best < 0 ? 0.f : score[best];
            if (lane == 0) {
                ids[(size_t)n * top + j] = best < 0 ? 0 : best;
                weights[(size_t)n * top + j] = wj;
                if (best >= 0) choice[best] = -INFINITY;  // taken
            }
            total += wj;
            __syncwarp();
        }
    } else {
        // softmax over all experts (lanes share the work, every lane ends with the same numbers)
        float m = -INFINITY;
        for (int e = lane; e < experts; e += 32) m = fmaxf(m, score[e]);
        m = warp_max(m);
        float sum = 0.f;
        for (int e = lane; e < experts; e += 32) {
            float p = expf(score[e] - m);
            score[e] = p;
            sum += p;
        }
        sum = warp_sum(sum);
        float inv = 1.0f / sum;
        for (int e = lane; e < experts; e += 32) score[e] *= inv;
        __syncwarp();
        // keep the best groups: a group that is not kept gets its experts' scores hidden (negated - 1)
        if (keep < groups) {
            for (int g = lane; g < groups; g += 32) {
                float b = -1.f;
                for (int e = g * per; e < (g + 1) * per; ++e) b = fmaxf(b, score[e]);
                gbest[g] = b;
            }
            __syncwarp();
            for (int round = 0; round < keep; ++round) {
                const int best = warp_best(gbest, groups, -1.f, lane);
                if (best < 0) break;
                if (lane == 0) gbest[best] = -2.f - gbest[best];  // marked as kept
                __syncwarp();
            }
            for (int e = lane; e < experts; e += 32)
                if (gbest[e / per] >= 0.f) score[e] = -1.f - score[e];
            __syncwarp();
        }
        for (int j = 0; j < top; ++j) {
            const int best = max(warp_best(score, experts, -1e-30f, lane), 0);
            const float s = score[best], bv = s >= 0.f ? s : 0.f;  // (no score to choose: expert 0 without weight)
            __syncwarp();
            if (lane == 0) {
                ids[(size_t)n * top + j] = best;
                weights[(size_t)n * top + j] = bv;
                score[best] = -1.f - s;  // taken
            }
            total += bv;
            __syncwarp();
        }
    }
    const float f = weight_scale / (total + 1e-20f);
    if (lane == 0)
        for (int j = 0; j < top; ++j) weights[(size_t)n * top + j] *= f;
}

// TOKENS tokens per block: the router's rows are read once for all of them.  A token at a time 2,048 tokens of width 2,048 with 32
// experts read them 2,048 times (half a GB through the L2, 47 us); few tokens want a block each.  What bounds it is the way to the
// L2 and back, so a lane has eight pieces of the router's rows on their way, the first of them before the tokens' own rows have arrived,
// and the choice is the whole warp's (8 tokens, 32 experts: 20 -> 11 us).
// A step of no more tokens than SMs takes blocks of 1,024 threads, one an SM; one of two, three or four times as many blocks of 256, so many an SM, with
// fewer registers and so fewer loads ahead each: all blocks run at one time.  (With 1,024 threads every further 148 tokens are another round.  2,048
// wide, 32 experts, us with them / so: 148 tokens 6.9 / 6.9, 160 12.6 / 7.7, 300 18.7 / 9.0, 500 25.6 / 11.9; 1,024 wide, 16 experts, 500 17.4 / 7.7.)
template <typename T, int TOKENS, int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS)
route_topk_kernel(const T* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, int num_tokens, int width,
                  int experts, int top, int groups, int keep, int sigmoid_scores,
                  const float* __restrict__ correction, int group_top, float weight_scale, int whole_pieces,
                  int* __restrict__ ids, float* __restrict__ weights) {
    extern __shared__ __align__(16) float sm[];  // x[TOKENS][width], then per token score[experts], group_best[groups], choice[experts]
    float* xs = sm;
    const int n0 = blockIdx.x * TOKENS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cnt = min(TOKENS, num_tokens - n0);
    float* const scores = xs + TOKENS * width;
    const int per_token = 2 * experts + groups;
    // A warp takes every so many'th expert, some of them at a time.  An expert's sum is the same chain of operations whichever
    // way it is grouped: four partial sums per lane, added in a fixed order.
    constexpr int WARPS = THREADS / 32, AT_ONCE = THREADS > 256 ? 1 : 4, AHEAD = BLOCKS == 1 ? 8 : BLOCKS == 2 ? 2 : 1;
    float4 wv[AHEAD][AT_ONCE];
    auto ask = [&](int slot, int e0, int i) {
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            const int e = e0 + u * WARPS;
            wv[slot][u] = e < experts && i < width ? *reinterpret_cast<const float4*>(w + (size_t)e * width + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto ask_first = [&](int e0) {
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) ask(a, e0, lane * 4 + a * 128);
    };
    ie_pdl_trigger();
    if (width % 4 == 0) ask_first(warp);  // (weights: nothing that the kernel before writes)
    ie_pdl_wait();
    if (whole_pieces) {  // rows of whole 16-byte pieces, aligned
        constexpr int PIECE = 16 / sizeof(T);
        for (int i = tid * PIECE; i < TOKENS * width; i += THREADS * PIECE) {
            float4 v[PIECE / 4];
            if (i < cnt * width) {
                const uint4 raw = *reinterpret_cast<const uint4*>(x + (size_t)n0 * width + i);
                const T* t = reinterpret_cast<const T*>(&raw);
#pragma unroll
                for (int k = 0; k < PIECE / 4; ++k)
                    v[k] = make_float4(ie_load(t + 4 * k), ie_load(t + 4 * k + 1), ie_load(t + 4 * k + 2), ie_load(t + 4 * k + 3));
            } else {
#pragma unroll
                for (int k = 0; k < PIECE / 4; ++k) v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < PIECE / 4; ++k) *reinterpret_cast<float4*>(xs + i + 4 * k) = v[k];
        }
    } else {
        for (int i = tid; i < TOKENS * width; i += THREADS) xs[i] = i < cnt * width ? ie_load(x + (size_t)n0 * width + i) : 0.f;
    }
    __syncthreads();
    for (int e0 = warp; e0 < experts; e0 += WARPS * AT_ONCE) {
        float acc[AT_ONCE][TOKENS];
        if (width % 4 == 0) {
            float a4[AT_ONCE][TOKENS][4];
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u)
#pragma unroll
                for (int t = 0; t < TOKENS; ++t) a4[u][t][0] = a4[u][t][1] = a4[u][t][2] = a4[u][t][3] = 0.f;
            if (e0 != warp) ask_first(e0);
            for (int i0 = lane * 4; i0 < width; i0 += 128 * AHEAD) {
#pragma unroll
                for (int a = 0; a < AHEAD; ++a) {
                    const int i = i0 + a * 128;
                    if (i < width) {
#pragma unroll
                        for (int t = 0; t < TOKENS; ++t) {
                            float4 xv = *reinterpret_cast<const float4*>(xs + t * width + i);
#pragma unroll
                            for (int u = 0; u < AT_ONCE; ++u) {
                                a4[u][t][0] = fmaf(xv.x, wv[a][u].x, a4[u][t][0]); a4[u][t][1] = fmaf(xv.y, wv[a][u].y, a4[u][t][1]);
                                a4[u][t][2] = fmaf(xv.z, wv[a][u].z, a4[u][t][2]); a4[u][t][3] = fmaf(xv.w, wv[a][u].w, a4[u][t][3]);
                            }
                        }
                        ask(a, e0, i + 128 * AHEAD);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u)
#pragma unroll
                for (int t = 0; t < TOKENS; ++t) acc[u][t] = (a4[u][t][0] + a4[u][t][1]) + (a4[u][t][2] + a4[u][t][3]);
        } else {
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) {
                int e = e0 + u * WARPS;
#pragma unroll
                for (int t = 0; t < TOKENS; ++t) {
                    acc[u][t] = 0.f;
                    if (e < experts)
                        for (int i = lane; i < width; i += 32) acc[u][t] = fmaf(xs[t * width + i], w[(size_t)e * width + i], acc[u][t]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) {
            int e = e0 + u * WARPS;
#pragma unroll
            for (int t = 0; t < TOKENS; ++t) {
                float total = warp_sum(acc[u][t]);
                if (lane == 0 && e < experts) scores[t * per_token + e] = bias != nullptr ? total + bias[e] : total;
            }
        }
    }
    __syncthreads();
    if (warp >= cnt) return;  // (a warp per token from here on)
    float* score = scores + warp * per_token;
    choose_experts(n0 + warp, score, score + experts, score + experts + groups, lane, experts, top, groups, keep, sigmoid_scores, correction,
                   group_top, weight_scale, ids, weights);
}

// The same for many bfloat16 tokens: 16 a block, whose products with the router's rows run on the tensor cores.  A 32-bit number is a sum of
// three bfloat16 ones, so a product with a bfloat16 number is the sum of three that the tensor cores take whole; 16 of k go through them, whose
// sums cut off what does not fit, and are added in 32 bits.  A warp takes every sixteenth 32 of k, and the warps' sums meet by halves of them, which
// leaves less error than one after the other: weights against 64 bits, 2,048 tokens of width 2,048 with 32-bit router rows 1.50e-7 by chains, 1.78e-7
// by 32 of k and one warp after the other, 1.41e-7 so; with router rows of bfloat16 numbers 1.37e-7, 1.55e-7 and 1.37e-7.
// (2,048 tokens of width 2,048, 32 experts: 41 us by multiply-adds, four tokens a block, bound by the router's rows' way from the L2; 21 us
// with eight warps, 14 with sixteen.)
constexpr int RM_TOKENS = 16, RM_WARPS = 16, RM_EXPERTS = 32;

__device__ __forceinline__ void three(float x, float y, unsigned (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
        t[i] = *reinterpret_cast<const unsigned*>(&v);
        if (i < 2) {
            x -= __uint_as_float(t[i] << 16);
            y -= __uint_as_float(t[i] & 0xFFFF0000u);
        }
    }
}

// One chain of multiply-adds: for a logit that is no finite number, which three parts, added up or multiplied with an infinite value, do not keep as it is.
__device__ __noinline__ float route_chain(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, int width) {
    float s = 0.f;
#pragma unroll 4
    for (int k = 0; k < width; ++k) s = fmaf(__bfloat162float(x[k]), w[k], s);
    return s;
}

__global__ void __launch_bounds__(RM_WARPS * 32)
route_many_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias, int num_tokens, int width,
                  int experts, int top, int groups, int keep, int sigmoid_scores, const float* __restrict__ correction, int group_top,
                  float weight_scale, int* __restrict__ ids, float* __restrict__ weights) {
    extern __shared__ __align__(16) float sm[];  // [16 warps][16 tokens][33], then per token score[experts], group_best[groups], choice[experts]
    constexpr int LD = RM_EXPERTS + 1;
    float* const scores = sm + RM_WARPS * RM_TOKENS * LD;
    const int per_token = 2 * experts + groups;
    const int n0 = blockIdx.x * RM_TOKENS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    ie_pdl_trigger();
    ie_pdl_wait();
    // the lane's eight k of 32: two instructions' worth, in an order of its own that both factors share
    const uint4* x0 = reinterpret_cast<const uint4*>(x + (size_t)min(n0 + g, num_tokens - 1) * width) + t;
    const uint4* x1 = reinterpret_cast<const uint4*>(x + (size_t)min(n0 + 8 + g, num_tokens - 1) * width) + t;
    for (int e0 = 0; e0 < experts; e0 += RM_EXPERTS) {
        float acc[4][4] = {};
        uint4 a0, a1;
        float4 wv[4][2];
        auto ask = [&](int k) {
            if (k >= width) return;
            a0 = x0[k / 8];
            a1 = x1[k / 8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int e = e0 + 8 * j + g;
                const float4* p = reinterpret_cast<const float4*>(w + (size_t)e * width + k + 8 * t);
                wv[j][0] = e < experts ? p[0] : make_float4(0.f, 0.f, 0.f, 0.f);
                wv[j][1] = e < experts ? p[1] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        ask(warp * 32);
        for (int k = warp * 32; k < width; k += RM_WARPS * 32) {
            const unsigned av[2][4] = {{a0.x, a1.x, a0.y, a1.y}, {a0.z, a1.z, a0.w, a1.w}};
            unsigned b[4][2][2][3];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    three(wv[j][h].x, wv[j][h].y, b[j][h][0]);
                    three(wv[j][h].z, wv[j][h].w, b[j][h][1]);
                }
            ask(k + RM_WARPS * 32);  // (the next ones are on their way during the products)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float c[2][4] = {};  // 16 of k each, lower parts first, so that little is cut off
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 2; i >= 0; --i)
                        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                            : "+f"(c[h][0]), "+f"(c[h][1]), "+f"(c[h][2]), "+f"(c[h][3])
                            : "r"(av[h][0]), "r"(av[h][1]), "r"(av[h][2]), "r"(av[h][3]), "r"(b[j][h][0][i]), "r"(b[j][h][1][i]));
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[j][i] += c[0][i] + c[1][i];
            }
        }
        float* mine = sm + warp * RM_TOKENS * LD;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) mine[(g + 8 * (i >> 1)) * LD + 8 * j + 2 * t + (i & 1)] = acc[j][i];
        __syncthreads();
        for (int i = tid; i < RM_TOKENS * RM_EXPERTS; i += RM_WARPS * 32) {
            const int row = i / RM_EXPERTS, e = e0 + i % RM_EXPERTS;
            if (e < experts) {
                float part[RM_WARPS];  // the warps' sums, by halves of them
#pragma unroll
                for (int v = 0; v < RM_WARPS; ++v) part[v] = sm[(v * RM_TOKENS + row) * LD + i % RM_EXPERTS];
#pragma unroll
                for (int half = RM_WARPS / 2; half > 0; half >>= 1)
#pragma unroll
                    for (int v = 0; v < half; ++v) part[v] += part[v + half];
                float s = part[0];
                if (!isfinite(s) && n0 + row < num_tokens) s = route_chain(x + (size_t)(n0 + row) * width, w + (size_t)e * width, width);
                scores[row * per_token + e] = bias != nullptr ? s + bias[e] : s;
            }
        }
        __syncthreads();
    }
    for (int row = warp; row < min(RM_TOKENS, num_tokens - n0); row += RM_WARPS) {
        float* score = scores + row * per_token;
        choose_experts(n0 + row, score, score + experts, score + experts + groups, lane, experts, top, groups, keep, sigmoid_scores, correction,
                       group_top, weight_scale, ids, weights);
    }
}

constexpr int TILE_M = 64, TILE_N = 64, TILE_K = 32;

// sorted[tiles * TILE_M]: pair index (token * top + choice) or -1; tile_expert[tiles]; meta[0] = tiles.
__global__ void __launch_bounds__(1024)
routed_align_kernel(const int* __restrict__ ids, int pairs, int experts, int* __restrict__ sorted,
                    int* __restrict__ tile_expert, int* __restrict__ meta, int max_tiles) {
    extern __shared__ int ism[];  // count[experts], first[experts] (first row of the expert's run), cursor[experts]
    int* count = ism;
    int* first = count + experts;
    int* cursor = first + experts;
    ie_pdl_trigger();
    ie_pdl_wait();
    int tid = threadIdx.x;
    for (int e = tid; e < experts; e += blockDim.x) { count[e] = 0; cursor[e] = 0; }
    for (int i = tid; i < max_tiles * TILE_M; i += blockDim.x) sorted[i] = -1;
    __syncthreads();
    for (int i = tid; i < pairs; i += blockDim.x) {
        int e = ids[i];
        if (e >= 0 && e < experts) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    if (tid == 0) {
        int tiles = 0;
        for (int e = 0; e < experts; ++e) {
            first[e] = tiles * TILE_M;
            int t = (count[e] + TILE_M - 1) / TILE_M;
            for (int j = 0; j < t && tiles + j < max_tiles; ++j) tile_expert[tiles + j] = e;
            tiles += t;
        }
        meta[0] = tiles < max_tiles ? tiles : max_tiles;
    }
    __syncthreads();
    for (int i = tid; i < pairs; i += blockDim.x) {
        int e = ids[i];
        if (e < 0 || e >= experts) continue;
        int at = first[e] + atomicAdd(&cursor[e], 1);
        if (at < max_tiles * TILE_M) sorted[at] = i;
    }
}

// ---- tile products -----------------------------------------------------------------------------
// A tile: up to TILE_M rows (given by pointers, nullptr = a padding row of zeros) times TILE_N rows
// of a [*, K] matrix, over all of K.  128 threads.

// 32-bit: thread (ty, tx) of 8 x 16 owns rows ty*8 .. +7 and columns tx*4 .. +3.
struct TileF32 {
    static constexpr int ACC = 32;
    float (*as)[TILE_M + 4];
    float (*bs)[TILE_N + 4];
    __device__ void zero(float* acc) {
#pragma unroll
        for (int i = 0; i < ACC; ++i) acc[i] = 0.f;
    }
    __device__ void load_a(const float* const* rows, int k0, int K) {
        for (int i = threadIdx.x; i < TILE_M * TILE_K; i += 128) {
            int r = i / TILE_K, k = i - r * TILE_K;
            const float* p = rows[r];
            as[k][r] = (p != nullptr && k0 + k < K) ? p[k0 + k] : 0.f;
        }
    }
    __device__ void load_b(const float* w, int n0, int N, int k0, int K) {
        for (int i = threadIdx.x; i < TILE_N * TILE_K; i += 128) {
            int r = i / TILE_K, k = i - r * TILE_K;
            bs[k][r] = (n0 + r < N && k0 + k < K) ? w[(size_t)(n0 + r) * K + k0 + k] : 0.f;
        }
    }
    __device__ void mma(float* acc) {
        int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll
        for (int k = 0; k < TILE_K; ++k) {
            float a[8], b[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = as[k][ty * 8 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = bs[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i * 4 + j] = fmaf(a[i], b[j], acc[i * 4 + j]);
        }
    }
    // element e of a thread's accumulators -> (row, column) inside the tile
    __device__ static void where(int e, int& r, int& c) {
        r = (threadIdx.x >> 4) * 8 + e / 4;
        c = (threadIdx.x & 15) * 4 + e % 4;
    }
};

// bfloat16: warp w of 4 owns rows (w >> 1) * 32 .. +31 and columns (w & 1) * 32 .. +31: two 16-row
// and four 8-column instruction tiles.
struct TileBF16 {
    static constexpr int ACC = 32;
    static constexpr int LD = TILE_K + 8;  // bfloat16 per shared-memory row (80 bytes: no bank conflicts)
    __nv_bfloat16 (*as)[LD];
    __nv_bfloat16 (*bs)[LD];
    __device__ void zero(float* acc) {
#pragma unroll
        for (int i = 0; i < ACC; ++i) acc[i] = 0.f;
    }
    __device__ static void load_rows(__nv_bfloat16 (*dst)[LD], int r, int seg, const __nv_bfloat16* p, int k0, int K, bool vec) {
        // 8 entries (16 bytes) of row r from column k0 + seg * 8
        int k = k0 + seg * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (p != nullptr) {
            if (vec && k + 8 <= K) v = *reinterpret_cast<const uint4*>(p + k);
            else {
                __nv_bfloat16 tmp[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) tmp[i] = (k + i < K) ? p[k + i] : __float2bfloat16_rn(0.f);
                v = *reinterpret_cast<uint4*>(tmp);
            }
        }
        *reinterpret_cast<uint4*>(&dst[r][seg * 8]) = v;
    }
    __device__ void load_a(const __nv_bfloat16* const* rows, int k0, int K) {
        bool vec = (K % 8 == 0);
        for (int i = threadIdx.x; i < TILE_M * (TILE_K / 8); i += 128) {
            int r = i >> 2, seg = i & 3;
            load_rows(as, r, seg, rows[r], k0, K, vec);
        }
    }
    __device__ void load_b(const __nv_bfloat16* w, int n0, int N, int k0, int K) {
        bool vec = (K % 8 == 0);
        for (int i = threadIdx.x; i < TILE_N * (TILE_K / 8); i += 128) {
            int r = i >> 2, seg = i & 3;
            load_rows(bs, r, seg, n0 + r < N ? w + (size_t)(n0 + r) * K : nullptr, k0, K, vec);
        }
    }
    __device__ void mma(float* acc) {
        int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        int rm = (warp >> 1) * 32, cn = (warp & 1) * 32;
#pragma unroll
        for (int kk = 0; kk < TILE_K; kk += 16) {
            unsigned a[2][4], b[4][2];
            // A: a 16 x 16 tile per x4; B: two 8-column tiles (both halves of k) per x4
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) {
                unsigned addr = (unsigned)__cvta_generic_to_shared(&as[rm + mi * 16 + (lane & 15)][kk + (lane >> 4) * 8]);
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                             : "=r"(a[mi][0]), "=r"(a[mi][1]), "=r"(a[mi][2]), "=r"(a[mi][3]) : "r"(addr));
            }
#pragma unroll
            for (int nj = 0; nj < 4; nj += 2) {
                unsigned addr = (unsigned)__cvta_generic_to_shared(
                    &bs[cn + nj * 8 + (lane & 7) + ((lane >> 4) & 1) * 8][kk + ((lane >> 3) & 1) * 8]);
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                             : "=r"(b[nj][0]), "=r"(b[nj][1]), "=r"(b[nj + 1][0]), "=r"(b[nj + 1][1]) : "r"(addr));
            }
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) {
                    float* c = acc + (mi * 4 + ni) * 4;
                    asm volatile(
                        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                        : "r"(a[mi][0]), "r"(a[mi][1]), "r"(a[mi][2]), "r"(a[mi][3]), "r"(b[ni][0]), "r"(b[ni][1]));
                }
        }
    }
    __device__ static void where(int e, int& r, int& c) {
        int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        int mi = e / 16, ni = (e / 4) % 4, j = e % 4;
        r = (warp >> 1) * 32 + mi * 16 + (lane >> 2) + (j >> 1) * 8;
        c = (warp & 1) * 32 + ni * 8 + (lane & 3) * 2 + (j & 1);
    }
};

template <typename T> struct TileOf;
template <> struct TileOf<float> { using type = TileF32; };
template <> struct TileOf<__nv_bfloat16> { using type = TileBF16; };

template <typename T>
__device__ __forceinline__ typename TileOf<T>::type make_tile(unsigned char* raw) {
    typename TileOf<T>::type tile;
    if constexpr (sizeof(T) == 4) {
        tile.as = reinterpret_cast<float (*)[TILE_M + 4]>(raw);
        tile.bs = reinterpret_cast<float (*)[TILE_N + 4]>(raw + sizeof(float) * TILE_K * (TILE_M + 4));
    } else {
        tile.as = reinterpret_cast<__nv_bfloat16 (*)[TileBF16::LD]>(raw);
        tile.bs = reinterpret_cast<__nv_bfloat16 (*)[TileBF16::LD]>(raw + sizeof(__nv_bfloat16) * TILE_M * TileBF16::LD);
    }
    return tile;
}

constexpr size_t TILE_SMEM_F32 = sizeof(float) * TILE_K * (TILE_M + 4 + TILE_N + 4);
constexpr size_t TILE_SMEM = TILE_SMEM_F32;  // the bfloat16 tiles need less

// x: [N, K]; w_gate_up: [experts, 2, F, K]; y: [pairs, F].
template <typename T>
__global__ void __launch_bounds__(128)
routed_gate_up_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y,
                      const int* __restrict__ sorted, const int* __restrict__ tile_expert,
                      const int* __restrict__ meta, int top, int K, int F, float limit, int clamp,
                      float alpha, float up_offset) {
    __shared__ __align__(16) unsigned char raw[TILE_SMEM];
    __shared__ const T* rows[TILE_M];
    __shared__ int pair_of[TILE_M];
    ie_pdl_trigger();
    ie_pdl_wait();
    int tile_id = blockIdx.y;
    if (tile_id >= meta[0]) return;
    int e = tile_expert[tile_id], n0 = blockIdx.x * TILE_N;
    if (threadIdx.x < TILE_M) {
        int pair = sorted[tile_id * TILE_M + threadIdx.x];
        pair_of[threadIdx.x] = pair;
        rows[threadIdx.x] = pair >= 0 ? x + (size_t)(pair / top) * K : nullptr;
    }
    __syncthreads();
    auto tile = make_tile<T>(raw);
    const T* wg = w + (size_t)e * 2 * F * K;
    const T* wu = wg + (size_t)F * K;
    float gate[32], up[32];
    tile.zero(gate);
    tile.zero(up);
    for (int k0 = 0; k0 < K; k0 += TILE_K) {
        tile.load_a(rows, k0, K);
        tile.load_b(wg, n0, F, k0, K);
        __syncthreads();
        tile.mma(gate);
        __syncthreads();
        tile.load_b(wu, n0, F, k0, K);
        __syncthreads();
        tile.mma(up);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        int r, c;
        tile.where(i, r, c);
        int pair = pair_of[r];
        if (pair < 0 || n0 + c >= F) continue;
        float g = gate[i], u = up[i];
        if (clamp) { g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit); }
        float act = g / (1.0f + expf(-alpha * g)) * (u + up_offset);
        ie_store(y + (size_t)pair * F + n0 + c, act);
    }
}

// y: [pairs, F]; w_down: [experts, H, F]; out: [top, N, H] 32-bit.
template <typename T>
__global__ void __launch_bounds__(128)
routed_down_kernel(const T* __restrict__ y, const T* __restrict__ w, float* __restrict__ out,
                   const float* __restrict__ weights, const int* __restrict__ sorted,
                   const int* __restrict__ tile_expert, const int* __restrict__ meta, int top, int N,
                   int F, int H) {
    __shared__ __align__(16) unsigned char raw[TILE_SMEM];
    __shared__ const T* rows[TILE_M];
    __shared__ int pair_of[TILE_M];
    ie_pdl_trigger();
    ie_pdl_wait();
    int tile_id = blockIdx.y;
    if (tile_id >= meta[0]) return;
    int e = tile_expert[tile_id], n0 = blockIdx.x * TILE_N;
    if (threadIdx.x < TILE_M) {
        int pair = sorted[tile_id * TILE_M + threadIdx.x];
        pair_of[threadIdx.x] = pair;
        rows[threadIdx.x] = pair >= 0 ? y + (size_t)pair * F : nullptr;
    }
    __syncthreads();
    auto tile = make_tile<T>(raw);
    const T* wd = w + (size_t)e * H * F;
    float acc[32];
    tile.zero(acc);
    for (int k0 = 0; k0 < F; k0 += TILE_K) {
        tile.load_a(rows, k0, F);
        tile.load_b(wd, n0, H, k0, F);
        __syncthreads();
        tile.mma(acc);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        int r, c;
        tile.where(i, r, c);
        int pair = pair_of[r];
        if (pair < 0 || n0 + c >= H) continue;
        int token = pair / top, choice = pair - token * top;
        out[((size_t)choice * N + token) * H + n0 + c] = weights[pair] * acc[i];
    }
}

// ---- bfloat16 with rows that are multiples of 16 bytes: the same tiles fed by cp.async -------------
// Three stages of (rows of A, NB matrices' rows) in flight; one barrier per 32 columns of k.
// NB = 2: gate and up, then the activation; NB = 1: the down product, times the routing weight.
constexpr int PIPE_STAGES = 3;
constexpr int PIPE_LD = TileBF16::LD;
constexpr size_t pipe_smem(int nb) { return (size_t)PIPE_STAGES * (1 + nb) * TILE_M * PIPE_LD * sizeof(__nv_bfloat16); }

__device__ __forceinline__ void cp16(void* dst, const void* src, int bytes) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <int NB>
__global__ void __launch_bounds__(128)
routed_bf16_kernel(const __nv_bfloat16* __restrict__ a_rows, const __nv_bfloat16* __restrict__ w,
                   __nv_bfloat16* __restrict__ y, float* __restrict__ out, const float* __restrict__ weights,
                   const int* __restrict__ sorted, const int* __restrict__ tile_expert, const int* __restrict__ meta,
                   int top, int N, int K, int F, float limit, int clamp, float alpha, float up_offset) {
    // NB = 2: a_rows = x [N, K], w = [experts, 2, F, K], output y [pairs, F]
    // NB = 1: a_rows = y [pairs, K], w = [experts, F, K] (F = the model's width), output out [top, N, F]
    extern __shared__ __align__(16) unsigned char pipe_raw[];
    __shared__ const __nv_bfloat16* rows[TILE_M];
    __shared__ int pair_of[TILE_M];
    ie_pdl_trigger();
    ie_pdl_wait();
    int tile_id = blockIdx.y;
    if (tile_id >= meta[0]) return;
    int e = tile_expert[tile_id], n0 = blockIdx.x * TILE_N;
    if (threadIdx.x < TILE_M) {
        int pair = sorted[tile_id * TILE_M + threadIdx.x];
        pair_of[threadIdx.x] = pair;
        rows[threadIdx.x] = pair < 0 ? nullptr : a_rows + (size_t)(NB == 2 ? pair / top : pair) * K;
    }
    __syncthreads();
    auto stage_ptr = [&](int stage, int which) {
        return reinterpret_cast<__nv_bfloat16(*)[PIPE_LD]>(
            pipe_raw + ((size_t)stage * (1 + NB) + which) * TILE_M * PIPE_LD * sizeof(__nv_bfloat16));
    };
    const __nv_bfloat16* wb[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) wb[b] = w + ((size_t)e * NB + b) * F * K;
    auto issue = [&](int it) {
        int stage = it % PIPE_STAGES, k0 = it * TILE_K;
        for (int i = threadIdx.x; i < TILE_M * (TILE_K / 8); i += 128) {
            int r = i >> 2, k = k0 + (i & 3) * 8;
            bool in_k = k < K;
            const __nv_bfloat16* ap = rows[r];
            cp16(&stage_ptr(stage, 0)[r][(i & 3) * 8], ap != nullptr && in_k ? ap + k : a_rows, ap != nullptr && in_k ? 16 : 0);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                bool ok = in_k && n0 + r < F;
                cp16(&stage_ptr(stage, 1 + b)[r][(i & 3) * 8], ok ? wb[b] + (size_t)(n0 + r) * K + k : w, ok ? 16 : 0);
            }
        }
    };
    float acc[NB][32];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[b][i] = 0.f;
    int iters = (K + TILE_K - 1) / TILE_K;
    for (int it = 0; it < PIPE_STAGES - 1; ++it) {
        if (it < iters) issue(it);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    TileBF16 tile;
    for (int it = 0; it < iters; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(PIPE_STAGES - 2) : "memory");
        __syncthreads();
        if (it + PIPE_STAGES - 1 < iters) issue(it + PIPE_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        int stage = it % PIPE_STAGES;
        tile.as = stage_ptr(stage, 0);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            tile.bs = stage_ptr(stage, 1 + b);
            tile.mma(acc[b]);
        }
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        int r, c;
        TileBF16::where(i, r, c);
        int pair = pair_of[r];
        if (pair < 0 || n0 + c >= F) continue;
        if constexpr (NB == 2) {
            float g = acc[0][i], u = acc[NB - 1][i];
            if (clamp) { g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit); }
            y[(size_t)pair * F + n0 + c] = __float2bfloat16_rn(g / (1.0f + expf(-alpha * g)) * (u + up_offset));
        } else {
            int token = pair / top, choice = pair - token * top;
            out[((size_t)choice * N + token) * F + n0 + c] = weights[pair] * acc[0][i];
        }
    }
}
}  // namespace

IE_API int ie_route_topk(const void* x, int dtype, const float* w, const float* bias, int num_tokens, int width,
                         int experts, int top, int groups, int keep, int sigmoid_scores, const float* correction,
                         int group_top, float weight_scale, int* ids, float* weights, void* stream) {
    if (num_tokens <= 0) return 0;
    if (experts < 1 || groups < 1 || experts % groups || top < 1 || top > experts) return (int)cudaErrorInvalidValue;
    if (group_top < 1 || group_top > 2 || (!sigmoid_scores && (correction != nullptr || group_top != 1)))
        return (int)cudaErrorInvalidValue;
    // (four tokens a block from as many blocks as the device has SMs on, where their rows fit)
    constexpr int MANY = 4;
    size_t one = (size_t)(width + 2 * experts + groups) * sizeof(float);
    if (one > 48 * 1024) return (int)cudaErrorInvalidValue;
    const bool many = num_tokens >= MANY * ie_sm_count() && MANY * one <= 48 * 1024;
    const size_t smem = many ? MANY * one : one;
    const dim3 grid(many ? (num_tokens + MANY - 1) / MANY : num_tokens);
    const int whole_pieces = width % (dtype == IE_BF16 ? 8 : 4) == 0 && ((uintptr_t)x & 15) == 0;
    cudaStream_t s = (cudaStream_t)stream;
    const int an_sm = (num_tokens + ie_sm_count() - 1) / ie_sm_count();
#define IE_ROUTE(T, TOKENS, THREADS, BLOCKS)                                                                             \
    return ie_launch(route_topk_kernel<T, TOKENS, THREADS, BLOCKS>, grid, dim3(THREADS), smem, s, (const T*)x, w, bias, num_tokens, \
                     width, experts, top, groups, keep, sigmoid_scores, correction, group_top, weight_scale, whole_pieces, ids, weights)
    if (dtype == IE_BF16) {
        // (16 tokens a block from as many tokens on as four a block fill the device with, and rows of whole 32s)
        const size_t scratch = (size_t)RM_WARPS * RM_TOKENS * (RM_EXPERTS + 1) + (size_t)RM_TOKENS * (2 * experts + groups);
        if (num_tokens >= MANY * ie_sm_count() && width % 32 == 0 && whole_pieces && !((uintptr_t)w & 15) && scratch * sizeof(float) <= 48 * 1024)
            return ie_launch(route_many_kernel, dim3((num_tokens + RM_TOKENS - 1) / RM_TOKENS), dim3(RM_WARPS * 32), scratch * sizeof(float), s,
                             (const __nv_bfloat16*)x, w, bias, num_tokens, width, experts, top, groups, keep, sigmoid_scores, correction,
                             group_top, weight_scale, ids, weights);
        if (many) IE_ROUTE(__nv_bfloat16, MANY, 256, 2);
        if (an_sm <= 1) IE_ROUTE(__nv_bfloat16, 1, 1024, 1);
        if (an_sm <= 2) IE_ROUTE(__nv_bfloat16, 1, 256, 2);
        if (an_sm == 3) IE_ROUTE(__nv_bfloat16, 1, 256, 3);
        IE_ROUTE(__nv_bfloat16, 1, 256, 4);
    }
    if (many) IE_ROUTE(float, MANY, 256, 2);
    // (32-bit tokens a block of 1,024 each whatever their number: the products behind start early, and beside smaller blocks more of theirs meet on one SM
    // than pays.  The layer, 16 experts of 1,024 x 512, us with 256 / 1,024 threads: 200 tokens 548 / 528, 300 590 / 565, 450 642 / 604)
    IE_ROUTE(float, 1, 1024, 1);
#undef IE_ROUTE
}

IE_API int ie_routed_tile_rows() { return TILE_M; }

// The most tiles `pairs` pairs over `experts` experts can need.
IE_API int ie_routed_max_tiles(int pairs, int experts) {
    int used = pairs < experts ? pairs : experts;
    return pairs / TILE_M + used;
}

IE_API int ie_routed_align(const int* ids, int pairs, int experts, int* sorted, int* tile_expert, int* meta,
                           int max_tiles, void* stream) {
    if (pairs <= 0) return 0;
    size_t smem = (size_t)3 * experts * sizeof(int);
    if (smem > 48 * 1024) return (int)cudaErrorInvalidValue;
    return ie_launch(routed_align_kernel, dim3(1), dim3(1024), smem, (cudaStream_t)stream, ids, pairs, experts,
                     sorted, tile_expert, meta, max_tiles);
}

IE_API int ie_routed_gate_up(const void* x, const void* w, void* y, int dtype, const int* sorted,
                             const int* tile_expert, const int* meta, int max_tiles, int top, int K, int F,
                             float limit, int clamp, float alpha, float up_offset, void* stream) {
    if (max_tiles <= 0) return 0;
    dim3 grid((F + TILE_N - 1) / TILE_N, max_tiles);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == IE_BF16 && K % 8 == 0)
        return ie_launch(routed_bf16_kernel<2>, grid, dim3(128), pipe_smem(2), s, (const __nv_bfloat16*)x,
                         (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (float*)nullptr, (const float*)nullptr, sorted,
                         tile_expert, meta, top, 0, K, F, limit, clamp, alpha, up_offset);
    if (dtype == IE_BF16)
        return ie_launch(routed_gate_up_kernel<__nv_bfloat16>, grid, dim3(128), 0, s, (const __nv_bfloat16*)x,
                         (const __nv_bfloat16*)w, (__nv_bfloat16*)y, sorted, tile_expert, meta, top, K, F, limit,
                         clamp, alpha, up_offset);
    return ie_launch(routed_gate_up_kernel<float>, grid, dim3(128), 0, s, (const float*)x, (const float*)w,
                     (float*)y, sorted, tile_expert, meta, top, K, F, limit, clamp, alpha, up_offset);
}

IE_API int ie_routed_down(const void* y, const void* w, float* out, const float* weights, int dtype,
                          const int* sorted, const int* tile_expert, const int* meta, int max_tiles, int top,
                          int N, int F, int H, void* stream) {
    if (max_tiles <= 0) return 0;
    dim3 grid((H + TILE_N - 1) / TILE_N, max_tiles);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == IE_BF16 && F % 8 == 0)
        return ie_launch(routed_bf16_kernel<1>, grid, dim3(128), pipe_smem(1), s, (const __nv_bfloat16*)y,
                         (const __nv_bfloat16*)w, (__nv_bfloat16*)nullptr, out, weights, sorted, tile_expert, meta,
                         top, N, F, H, 0.f, 0, 0.f, 0.f);
    if (dtype == IE_BF16)
        return ie_launch(routed_down_kernel<__nv_bfloat16>, grid, dim3(128), 0, s, (const __nv_bfloat16*)y,
                         (const __nv_bfloat16*)w, out, weights, sorted, tile_expert, meta, top, N, F, H);
    return ie_launch(routed_down_kernel<float>, grid, dim3(128), 0, s, (const float*)y, (const float*)w, out,
                     weights, sorted, tile_expert, meta, top, N, F, H);
}
