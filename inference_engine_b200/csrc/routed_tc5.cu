// The routed feed-forward's two grouped products on the fifth-generation tensor cores, bfloat16 in, 32-bit sums in tensor memory.
//
//  * routed_sort: the step's (token, choice) pairs in the order of their experts, and a list of tiles: up to so many neighbouring
//    pairs of one expert (256 for the kernels here), an expert's pairs in equal tiles.  With `align` 8 an expert's run and its tiles start at
//    multiples of 8 (for the kernels of routed_tiled.cu); the places between hold -1.
//  * routed_tc5<true>: per tile and 128 hidden features: gate and up products, then the activation, to y[place in the order].
//  * routed_tc5<false>: per tile and 256 output features: y times the expert's down matrix, times the pair's routing weight, to
//    out[choice][token][:].
//
// The operands' roles are swapped: features are the instruction's 128 rows (tensor-memory lanes), a tile's pairs its columns, so an
// expert's pairs are rounded up to 16 only and not to a tile of 128 rows (2,048 tokens x 4 choices over 32 experts: 256 +- 14 pairs
// each).  A block holds two accumulators of 128 features (gate and up, or two runs of output features) x 256 pairs, all of tensor memory: per 64
// of k 64 KB arrive for 2 x 128 x 256 x 64 products, 64 bytes a clock, where one accumulator would ask the L2 for 96.
//   warp 0, one thread: tiled copies of the weights (and of y, whose rows are neighbours) into a ring of 192 KB; one copy brings both
//   runs of features, one or two bring y's rows: the copy engine spends some 300 clocks on each, and with six copies of 8 and 16 KB per
//   64 of k it was what the tensor cores waited for (2,048 tokens, 32 experts of 2,048 x 1,024: 160 and 88 us for the two products);
//   warp 1, one thread: tcgen05.mma; tcgen05.commit hands the ring's slots back;
//   warps 2-9: gather x's rows by cp.async, swizzled by hand as the copies are, and afterwards read the accumulators.
// Every wait is bounded; a block that waits too long records IE_ERR_TIMEOUT, frees its tensor memory and leaves.
#include "tma.cuh"
#include <math.h>

using namespace ie_tma;

namespace {
constexpr int FEATURES = 128, MOST_PAIRS = 256, BK = 64;
constexpr int W_BYTES = FEATURES * BK * 2;  // 16 KB
constexpr int RING_BYTES = 192 * 1024, MOST_SLOTS = 6;
constexpr int WORKERS = 8, THREADS = (2 + WORKERS) * 32;
// Rows of x are announced when the next ones have been asked for: with three slots a later announcement would have to wait for
// the products that read the slot in between.
constexpr int LAG = 1;

struct __align__(8) Shared {
    unsigned long long full[MOST_SLOTS], empty[MOST_SLOTS], acc_done;
    unsigned tmem_base;
    int failed;
    int row_of[MOST_PAIRS];  // a pair's row of x, or of the output
    float weight_of[MOST_PAIRS];
};
constexpr size_t SMEM_BYTES = (size_t)RING_BYTES + sizeof(Shared) + 1024;

// Tensor maps of y with boxes of 64, 128 and 256 rows: a tile's rows, rounded up to 64, in one or two copies.
struct RowMaps {
    CUtensorMap by64, by128, by256;
};

__device__ __forceinline__ void cp16(unsigned dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// grid: (blocks of features, tiles).  tiles: (expert, first place, pairs, 0); meta[0]: how many there are.
// GATED: x [N, K], w [experts, 2, F, K], y [pairs, F].  Else: y [pairs, K] through y_maps, w [experts, F, K], out [top, N, F].
template <bool GATED>
__global__ void __launch_bounds__(THREADS, 1)
routed_tc5_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ RowMaps y_maps, const bf16* __restrict__ x,
                  bf16* __restrict__ y, float* __restrict__ out, const float* __restrict__ weights, const int* __restrict__ order,
                  const int4* __restrict__ tiles, const int* __restrict__ meta, int top, int N, int K, int F, float limit, int clamp,
                  float alpha, float up_offset, int* err) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    Shared* sh = reinterpret_cast<Shared*>(ring + RING_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ie_pdl_trigger();
    ie_pdl_wait();
    if ((int)blockIdx.y >= meta[0]) return;  // (the whole block, before any barrier)
    const int4 tile = tiles[blockIdx.y];
    const int n = tile.z, n_pad = (n + 15) & ~15;
    const int x_rows = (n + 63) & ~63, x_bytes = x_rows * BK * 2, slot_bytes = 2 * W_BYTES + x_bytes;
    const int slots = min(RING_BYTES / slot_bytes, MOST_SLOTS);  // at least 3
    const int nkb = (K + BK - 1) / BK;
    const int f0 = blockIdx.x * (GATED ? FEATURES : 2 * FEATURES);
    const bool both = GATED || f0 + FEATURES < F;

    if (threadIdx.x == 0) {
        for (int s = 0; s < slots; ++s) {
            mbar_init(&sh->full[s], GATED ? 1 + WORKERS : 1);
            mbar_init(&sh->empty[s], 1);
        }
        mbar_init(&sh->acc_done, 1);
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp >= 2) {
        const int c = threadIdx.x - 64;
        const int pair = c < n ? order[tile.y + c] : -1;
        const int token = pair / top, choice = pair - token * top;
        sh->row_of[c] = pair < 0 ? -1 : GATED ? token : choice * N + token;
        if (!GATED) sh->weight_of[c] = pair >= 0 ? weights[pair] : 0.f;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = sh->tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            const int bytes = 2 * W_BYTES + (GATED ? 0 : x_bytes);
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % slots;
                if (kb >= slots && !mbar_wait_compact(&sh->empty[s], ((kb / slots) - 1) & 1)) { sh->failed = 1; break; }
                unsigned char* at = ring + (size_t)s * slot_bytes;
                mbar_expect_tx(&sh->full[s], bytes);
                if (GATED) {
                    tma_load_3d(at, &w_map, kb * BK, f0, 2 * tile.x, &sh->full[s]);  // 128 gate rows, 128 up rows
                } else {
                    tma_load_3d(at, &w_map, kb * BK, f0, tile.x, &sh->full[s]);      // 256 rows (zeros beyond the expert's)
                    unsigned char* xs = at + 2 * W_BYTES;
                    if (x_rows == 256) {
                        tma_load_2d(xs, &y_maps.by256, kb * BK, tile.y, &sh->full[s]);
                    } else {
                        if (x_rows >= 128) tma_load_2d(xs, &y_maps.by128, kb * BK, tile.y, &sh->full[s]);
                        if (x_rows & 64)
                            tma_load_2d(xs + (x_rows & 128) * BK * 2, &y_maps.by64, kb * BK, tile.y + (x_rows & 128), &sh->full[s]);
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            const unsigned idesc = umma_idesc_bf16(FEATURES, n_pad);
            bool ok = true;
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % slots;
                if (!mbar_wait_compact(&sh->full[s], (kb / slots) & 1)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned w0 = smem_u32(ring + (size_t)s * slot_bytes), x0 = w0 + 2 * W_BYTES;
#pragma unroll
                for (int ks = 0; ks < BK / 16; ++ks) {
                    const unsigned more = kb > 0 || ks > 0 ? 1u : 0u;
                    const unsigned long long xd = umma_desc_sw128(x0 + ks * 32);
                    umma_ss(tmem, umma_desc_sw128(w0 + ks * 32), xd, idesc, more);
                    if (both) umma_ss(tmem + MOST_PAIRS, umma_desc_sw128(w0 + W_BYTES + ks * 32), xd, idesc, more);
                }
                umma_commit(&sh->empty[s]);
            }
            if (!ok) sh->failed = 1;
            umma_commit(&sh->acc_done);
        }
        __syncwarp();
    } else {
        const int worker = threadIdx.x - 64;
        if (GATED) {
            // x's rows: eight threads a row, 32 rows at a time
            const int chunk = worker & 7, r0 = worker >> 3;
            const bf16* src[MOST_PAIRS / 32];
#pragma unroll
            for (int p = 0; p < MOST_PAIRS / 32; ++p) {
                const int row = sh->row_of[r0 + 32 * p];
                src[p] = row >= 0 ? x + (size_t)row * K + chunk * 8 : nullptr;
            }
            const unsigned to = (unsigned)((r0 * 8 + (chunk ^ (r0 & 7))) * 16);  // (r0 + 32 p: the same place in its group of eight rows)
            auto announce = [&](int kb) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->full[kb % slots]);
            };
            bool ok = true;
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % slots;
                if (kb >= slots && !mbar_wait_compact(&sh->empty[s], ((kb / slots) - 1) & 1)) { ok = false; break; }
                const unsigned base = smem_u32(ring + (size_t)s * slot_bytes + 2 * W_BYTES) + to;
                const int bytes = kb * BK + chunk * 8 < K ? 16 : 0;  // (beyond K: zeros; K is a multiple of 8)
#pragma unroll
                for (int p = 0; p < MOST_PAIRS / 32; ++p)
                    if (src[p] != nullptr) cp16(base + p * 32 * 128, bytes ? src[p] + kb * BK : x, bytes);
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (kb >= LAG) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
                    announce(kb - LAG);
                }
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (ok)
                for (int late = max(nkb - LAG, 0); late < nkb; ++late) announce(late);
            if (!ok) sh->failed = 1;
        }
        const bool ok = mbar_wait_compact(&sh->acc_done, 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (ok && !sh->failed) {
            const int group = warp & 3, side = (warp - 2) >> 2;  // a warp reads the 32 lanes 32 (warp % 4) ..
            const unsigned taddr = tmem + ((unsigned)(group * 32) << 16);
            const int f = f0 + group * 32 + lane;
            for (int c0 = side * 16; c0 < n_pad; c0 += 32) {
                float a[16], b[16];
                tmem_ld16(a, taddr + c0);
                if (both) tmem_ld16(b, taddr + MOST_PAIRS + c0);
                if (GATED) {
                    if (f < F)
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            if (c0 + i < n) {
                                float g = a[i], u = b[i];
                                if (clamp) { g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit); }
                                y[(size_t)(tile.y + c0 + i) * F + f] = __float2bfloat16_rn(g / (1.0f + expf(-alpha * g)) * (u + up_offset));
                            }
                        }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        if (c0 + i < n) {
                            const float w = sh->weight_of[c0 + i];
                            float* dst = out + (size_t)sh->row_of[c0 + i] * F + f;
                            if (f < F) dst[0] = w * a[i];
                            if (both && f + FEATURES < F) dst[FEATURES] = w * b[i];
                        }
                    }
                }
            }
        }
        if (!ok) sh->failed = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    if (threadIdx.x == 0 && sh->failed) ie_report(err, IE_ERR_TIMEOUT, blockIdx.x, blockIdx.y);
}

// One block.  order[pairs, or more with the gaps]: the pairs by expert (an id outside the experts leaves its pair out); tiles as above; meta: how
// many tiles, how many places.  A pair's rank among its
// expert's comes from the counter it raises; up to KEPT pairs of a thread keep it in registers, the rest take theirs in a second pass.
constexpr int SORT_THREADS = 1024, KEPT = 8;
__global__ void __launch_bounds__(SORT_THREADS, 1)
routed_sort_kernel(const int* __restrict__ ids, int pairs, int experts, int* __restrict__ order, int4* __restrict__ tiles,
                   int* __restrict__ meta, int max_tiles, int most, int align, int places) {
    extern __shared__ int ism[];  // count[experts], first[experts], tile[experts]
    int* count = ism;
    int* first = count + experts;
    int* tile0 = first + experts;
    __shared__ int total_tiles, total_places;
    ie_pdl_trigger();
    ie_pdl_wait();
    const int tid = threadIdx.x;
    int mine[KEPT], rank[KEPT];
#pragma unroll
    for (int k = 0; k < KEPT; ++k) {
        const int i = tid + k * SORT_THREADS;
        mine[k] = i < pairs ? ids[i] : -1;
    }
    for (int e = tid; e < experts; e += SORT_THREADS) count[e] = 0;
    if (align > 1)
        for (int i = tid; i < places; i += SORT_THREADS) order[i] = -1;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KEPT; ++k)
        if (mine[k] >= 0 && mine[k] < experts) rank[k] = atomicAdd(&count[mine[k]], 1);
    if (pairs > KEPT * SORT_THREADS) {
        __syncthreads();  // the ranks that are kept are the lowest
        for (int i = tid + KEPT * SORT_THREADS; i < pairs; i += SORT_THREADS) {
            const int e = ids[i];
            if (e >= 0 && e < experts) atomicAdd(&count[e], 1);
        }
    }
    __syncthreads();
    if (tid < 32) {  // running sums of pairs and tiles over the experts, 32 at a time
        int at = 0, t = 0;  // (places and tiles so far)
        for (int e0 = 0; e0 < experts; e0 += 32) {
            const int e = e0 + tid, pairs_of = e < experts ? count[e] : 0, k = (pairs_of + most - 1) / most;
            const int c = (pairs_of + align - 1) / align * align;
            int sc = c, sk = k;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int uc = __shfl_up_sync(0xffffffffu, sc, o), uk = __shfl_up_sync(0xffffffffu, sk, o);
                if (tid >= o) { sc += uc; sk += uk; }
            }
            if (e < experts) {
                first[e] = at + sc - c;
                tile0[e] = t + sk - k;
            }
            at += __shfl_sync(0xffffffffu, sc, 31);
            t += __shfl_sync(0xffffffffu, sk, 31);
        }
        if (tid == 0) { total_tiles = t; total_places = at; }
    }
    __syncthreads();
    if (tid == 0) { meta[0] = min(total_tiles, max_tiles); meta[1] = total_places; }
    for (int e = tid; e < experts; e += SORT_THREADS) {
        const int c = count[e], k = (c + most - 1) / most, units = (c + align - 1) / align;
        for (int j = 0; j < k; ++j) {  // (equal tiles, the earlier ones a pair, or `align` of them, longer)
            const int each = units / k, more = units - each * k, at = (j * each + min(j, more)) * align;
            if (tile0[e] + j < max_tiles) tiles[tile0[e] + j] = make_int4(e, first[e] + at, min((each + (j < more ? 1 : 0)) * align, c - at), 0);
        }
    }
#pragma unroll
    for (int k = 0; k < KEPT; ++k)
        if (mine[k] >= 0 && mine[k] < experts) order[first[mine[k]] + rank[k]] = tid + k * SORT_THREADS;
    if (pairs > KEPT * SORT_THREADS) {
        __syncthreads();
        // (the pairs in registers hold the lowest ranks; the others take theirs from the top down)
        for (int i = tid + KEPT * SORT_THREADS; i < pairs; i += SORT_THREADS) {
            const int e = ids[i];
            if (e >= 0 && e < experts) order[first[e] + atomicSub(&count[e], 1) - 1] = i;
        }
    }
}

// `matrices` row-major matrices [rows, cols] one behind the other as a 3-D tensor map, boxes of 64 columns (128 bytes, swizzled) x
// box_rows x box_matrices; what lies outside a matrix reads as zero.
bool make_expert_map(CUtensorMap* map, const void* base, int matrices, int rows, int cols, int box_rows, int box_matrices) {
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return false;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)matrices};
    cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)rows * cols * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, (cuuint32_t)box_matrices};
    cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

// Whether the kernels take these sizes (hidden and intermediate width multiples of 8).
IE_API int ie_routed_tc5_ok(int hidden, int ff) { return encode_fn() != nullptr && hidden % 8 == 0 && ff % 8 == 0 && hidden > 0 && ff > 0; }

// The most tiles `pairs` pairs over `experts` experts can need.
IE_API int ie_routed_tc5_max_tiles(int pairs, int experts, int most) { return pairs / most + (pairs < experts ? pairs : experts); }

IE_API int ie_routed_tc5_most() { return MOST_PAIRS; }

// places: the length of `order` (with `align` > 1: room for the gaps).
IE_API int ie_routed_sort(const int* ids, int pairs, int experts, int* order, int* tiles, int* meta, int max_tiles, int most, int align,
                          int places, void* stream) {
    if (pairs <= 0) return 0;
    if (most < align || align < 1 || (long long)places < pairs + (align - 1ll) * (pairs < experts ? pairs : experts)) return (int)cudaErrorInvalidValue;
    const size_t smem = (size_t)3 * experts * sizeof(int);
    if (smem > 40 * 1024 || ((uintptr_t)tiles & 15)) return (int)cudaErrorInvalidValue;
    return ie_launch(routed_sort_kernel, dim3(1), dim3(SORT_THREADS), smem, (cudaStream_t)stream, ids, pairs, experts, order,
                     (int4*)tiles, meta, max_tiles, most, align, places);
}

// x: [N, K], w: [experts, 2, F, K], y: [pairs, F] in the order of the pairs.
IE_API int ie_routed_tc5_gate_up(const void* x, const void* w, void* y, const int* order, const int* tiles, const int* meta,
                                 int max_tiles, int experts, int top, int K, int F, float limit, int clamp, float alpha,
                                 float up_offset, int* err, void* stream) {
    if (max_tiles <= 0) return 0;
    if (!ie_routed_tc5_ok(K, F) || (((uintptr_t)x | (uintptr_t)w) & 15)) return (int)cudaErrorInvalidValue;
    CUtensorMap wm;
    if (!make_expert_map(&wm, w, 2 * experts, F, K, FEATURES, 2)) return (int)cudaErrorNotSupported;
    const RowMaps unused = {};
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, routed_tc5_kernel<true>, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    return ie_launch(routed_tc5_kernel<true>, dim3((F + FEATURES - 1) / FEATURES, max_tiles), dim3(THREADS), SMEM_BYTES,
                     (cudaStream_t)stream, wm, unused, (const bf16*)x, (bf16*)y, (float*)nullptr, (const float*)nullptr, order,
                     (const int4*)tiles, meta, top, 0, K, F, limit, clamp, alpha, up_offset, err);
}

// y: [pairs, F], w: [experts, H, F], out: [top, N, H] 32-bit.
IE_API int ie_routed_tc5_down(const void* y, const void* w, float* out, const float* weights, const int* order, const int* tiles,
                              const int* meta, int max_tiles, int experts, int top, int N, int F, int H, int* err, void* stream) {
    if (max_tiles <= 0) return 0;
    if (!ie_routed_tc5_ok(H, F) || (((uintptr_t)y | (uintptr_t)w) & 15)) return (int)cudaErrorInvalidValue;
    CUtensorMap wm;
    RowMaps ym;
    const long long pairs = (long long)N * top;
    if (!make_expert_map(&wm, w, experts, H, F, 2 * FEATURES, 1) || !make_map_bf16(&ym.by64, y, pairs, F, 64) ||
        !make_map_bf16(&ym.by128, y, pairs, F, 128) || !make_map_bf16(&ym.by256, y, pairs, F, 256))
        return (int)cudaErrorNotSupported;
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, routed_tc5_kernel<false>, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    return ie_launch(routed_tc5_kernel<false>, dim3((H + 2 * FEATURES - 1) / (2 * FEATURES), max_tiles), dim3(THREADS), SMEM_BYTES,
                     (cudaStream_t)stream, wm, ym, (const bf16*)nullptr, (bf16*)nullptr, out, weights, order, (const int4*)tiles, meta,
                     top, N, F, H, 0.f, 0, 0.f, 0.f, err);
}
