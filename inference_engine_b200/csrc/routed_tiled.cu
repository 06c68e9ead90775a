// The routed feed-forward's two grouped products on weights laid out in tiles, bfloat16 in, 32-bit sums:
//
//  * gate-up: per tile of pairs (neighbouring (token, choice) pairs of one expert) and some hidden features, gate and up products and the
//    activation;
//  * down: per tile of pairs and some output features, y times the expert's down matrix, times the pairs' weights, to out[choice][token][:].
//
// Operands lie in memory as the tensor cores read them: 64 of k by so many rows, 128 bytes a row, a row's 16-byte pieces turned by
// its number (the 128-byte swizzle).  The weights in tiles of 128 rows, 16 KB each, a tile's k blocks behind one another (gate and up rows
// of 64 features alternate in blocks of 8); the pairs' rows, and y, as [k block][place][64], an expert's places from a multiple of 8 on.  So every
// copy is one run of bytes.  What bounds these products is the copies: with plain matrices and tiled copies (boxes of 128 rows of 128 bytes) an SM's
// copy engine brings 45 bytes a clock from the L2, runs of bytes 60 to 65, and 64 of k ask for 64 in the time of their products.
//
// Many pairs (`pair`): two blocks of a cluster work on one tile (tcgen05 cta_group::2): 256 rows of weights are the instruction's rows, 128
// in each block's tensor memory, up to 320 pairs its columns (in equal halves above 256), each block copying half of them.  An expert's pairs are
// rounded up to 32 and an expert of a few more than 256 pairs still is one tile, whose weights are read once.  The blocks stay and take tile
// after tile (a cluster takes every so many'th), with two accumulators of 256 columns: while the epilogue's warps read one, the tensor
// cores fill the other, and the copies of the next tile's operands run ahead of both.  More than 256 pairs take both.  (2,048 tokens, 4 of 32 experts of
// 2,048 x 1,024 each: 119 + 59 us with an SM a tile on plain matrices, 85 + 47 so, where the weights' bytes and the products take 43 + 21.)
//   warp 0, one thread of each block: copies into a ring of six slots of 36 KB (more and smaller ones where tiles are smaller, as in steps of fewer than 257 tokens);
//   warp 1 of the first block, one thread: tcgen05.mma for both (tcgen05.commit hands slots back and accumulators over in both blocks);
//   warps 2-9: read the accumulator of their block.
// Both blocks' copies are told to the first one's barrier, which is what orders them before the products that read them; copies of rows of 1 and 2 KB
// of a tensor map can be (cta_group::2), runs of bytes cannot, and they are as fast.  (With a word of the second block's for each of its slots: layer of 2,048 tokens
// 192 us where nothing orders that word, 294 where it is released to the cluster, a microsecond a word, 193 so; of 65 tokens 90, 211 and 92.)
//
// Few tokens (`few`: up to 64, tiles of at most 64 pairs): a stream of weights.  128 rows a block and 72 KB of ring, three blocks an SM:
// all blocks of a step start at once and share the memory evenly, and what one waits for at its start and end the others use.  (256 rows and an SM's
// whole memory a block: 8 tokens over 32 experts of 2,048 x 1,024 were 160 blocks of 1 MB in two rounds of 148, 49 + 26 us; 28 + 10 so.)
// The down product's weights are asked for while the gated product still runs (whose blocks let the next kernel start once they have
// seen the sorted pairs, so those are there).
//
// How many pairs a tile may have (`most`) goes into the sort, and both kernels cut their memory for it.  A step's tokens alone do not bound it: a token
// that names an expert more than once (routing does where its scores are no numbers, or where the kept groups have too few experts) has as many
// pairs there.
//
// Every wait is bounded; a block that waits too long records IE_ERR_TIMEOUT, and it (both of a cluster) leaves.
#include "tma.cuh"
#include <math.h>

using namespace ie_tma;

namespace {
constexpr int ROWS = 128, MOST_COLS = 256, MOST_PAIRS = 320, BK = 64;  // (320: also in halves rounded up to 32)
constexpr int W_BYTES = ROWS * BK * 2, X_BYTES = MOST_PAIRS / 2 * BK * 2, RING_BYTES = 6 * (W_BYTES + X_BYTES), MOST_SLOTS = 12;
static_assert((MOST_PAIRS / 2 + 31) / 32 * 32 <= MOST_PAIRS / 2, "both halves of a tile fit a slot");
constexpr int WORKERS = 8, THREADS = (2 + WORKERS) * 32;

struct __align__(16) Shared {
    unsigned long long full[MOST_SLOTS], empty[MOST_SLOTS], acc_full[2], acc_empty[2];
    unsigned tmem_base;
    int failed;
    alignas(16) int row_of[2][MOST_COLS];  // (down) a pair's row of the output, and its weight
    float weight_of[2][MOST_COLS];
};
constexpr size_t SMEM_BYTES = (size_t)RING_BYTES + sizeof(Shared) + 1024;

// A tile's pairs are the columns of one accumulator or, above 256, in equal halves of two.
__device__ __forceinline__ int parts(int n) { return n > MOST_COLS ? 2 : 1; }
// The columns of each, rounded up to what the instruction takes.
__device__ __forceinline__ int columns(int n) { return ((n + parts(n) - 1) / parts(n) + 31) & ~31; }

// (Many pairs) the weights' tiles as rows of 2 KB, boxes of 8; the pairs' rows as rows of 1 KB (8 places), boxes of 16, 8, 4 and 2.
struct Maps {
    CUtensorMap w, x[4];
};

struct Args {
    const unsigned char* w;  // the weights' tiles
    const unsigned char* x;  // the pairs' rows (few, gate-up: the tokens' rows as they are)
    const int4* tiles;       // (expert, first place, pairs, 0)
    const int* count;        // how many tiles there are
    int max_tiles, feature_blocks;
    int places;              // rows of a k block of x, and of y
    int w_blocks, kbs;       // tiles of 128 rows per expert, k blocks
    int slots, slot_bytes;   // (many pairs) of the ring
    int most;                // pairs of a tile that there is room for
    int K, F;                // (few, gate-up) columns of x; features of the result
    bf16* y;
    float* out;
    const int* order;
    const float* weights;
    int top, N;
    float limit, alpha, up_offset;
    int clamp;
    int* err;
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The first block's copy of an object in shared memory.
__device__ __forceinline__ unsigned in_first(const void* p) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
// (Of tensor memory alone, which tcgen05's fences order around a relaxed arrival.)
__device__ __forceinline__ void arrive_at(unsigned cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// A wait for what both blocks do: once it is over, a last look that acquires from the cluster.  (Each look one that acquires: 147 us instead of 113.)
__device__ __forceinline__ bool warp_wait_cluster(unsigned long long* bar, int parity) {
    if (!warp_wait(bar, parity)) return false;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%0], %1;\n}" ::"r"(smem_u32(bar)), "r"(parity) : "memory");
    return true;
}
// A box of whole rows of a map into this block's shared memory, told to the first block's barrier.
__device__ __forceinline__ void load_pair(void* dst, const CUtensorMap* map, int row, unsigned first_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(0), "r"(row), "r"(first_bar) : "memory");
}
// A run of `kilobytes` (up to 31, even) rows of 1 KB from `row` on, in boxes of 16, 8, 4 and 2 of them.
__device__ __forceinline__ void load_rows(unsigned char* dst, const CUtensorMap (&maps)[4], int row, int kilobytes, unsigned first_bar) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (kilobytes & (16 >> i)) {
            load_pair(dst, &maps[i], row, first_bar);
            dst += (16 >> i) * 1024;
            row += 16 >> i;
        }
}
// A run of bytes into this block's shared memory.
__device__ __forceinline__ void load_run(void* dst, const void* src, int bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ const unsigned char* w_tile(const Args& in, int expert, int block, int kb) {
    return in.w + (((size_t)expert * in.w_blocks + block) * in.kbs + kb) * W_BYTES;
}
// (The special-function unit's exponential and reciprocal by themselves are off by 12 units in the last place at gates of -8 and by 70 at -50; with them
// 2,048 tokens, 32 experts of 2,048 x 1,024: layer 181 us, 187 so; 8 tokens 60.4 and 61.1.)
__device__ __forceinline__ float activated(const Args& in, float g, float u) {
    if (in.clamp) { g = fminf(g, in.limit); u = fminf(fmaxf(u, -in.limit), in.limit); }
    return g / (1.0f + expf(-in.alpha * g)) * (u + in.up_offset);
}
// Sixteen columns of gates (lanes with bit 3 clear) and their ups (set), of the places from `first` (a multiple of 8) on, n of them there, to feature f
// of y: a lane takes every second place.  (Features beyond the last: zeros, from zero weights.)
__device__ __forceinline__ void put_gated(const Args& in, const float (&a)[16], bool high, int first, int n, int f) {
    unsigned char* y = reinterpret_cast<unsigned char*>(in.y + ((size_t)(f >> 6) * in.places + first + (high ? 1 : 0)) * 64 + (f & 7));
    const unsigned piece = (unsigned)(((f >> 3) & 7) ^ (high ? 1 : 0)) << 4;  // turned by the place's number, whose last bit is the lane's
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        const float other = __shfl_xor_sync(0xffffffffu, high ? a[i] : a[i + 1], 8);
        const float v = activated(in, high ? other : a[i], high ? a[i + 1] : other);
        if (i + (high ? 1 : 0) < n) *reinterpret_cast<bf16*>(y + i * 128 + (piece ^ ((i & 6) << 4))) = __float2bfloat16_rn(v);
    }
}
// D = or += A B^T.  PAIR: D in both blocks' tensor memory, A and B half in each block's shared memory, issued in the first block.
template <bool PAIR>
__device__ __forceinline__ void mma(unsigned d, unsigned a, unsigned b, unsigned idesc, bool accumulate) {
    if (PAIR)
        asm volatile("{\n .reg .pred p;\n .reg .b64 x, y;\n setp.ne.b32 p, %5, 0;\n mov.b64 x, {%1, %3};\n mov.b64 y, {%2, %3};\n"
                     " tcgen05.mma.cta_group::2.kind::f16 [%0], x, y, %4, p;\n}"
                     ::"r"(d), "r"(a), "r"(b), "r"(UMMA_DESC_HIGH), "r"(idesc), "r"((unsigned)accumulate) : "memory");
    else
        asm volatile("{\n .reg .pred p;\n .reg .b64 x, y;\n setp.ne.b32 p, %5, 0;\n mov.b64 x, {%1, %3};\n mov.b64 y, {%2, %3};\n"
                     " tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %4, p;\n}"
                     ::"r"(d), "r"(a), "r"(b), "r"(UMMA_DESC_HIGH), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
// An arrival at the barrier of both blocks when all that this thread issued so far is done.
__device__ __forceinline__ void pair_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((unsigned short)3) : "memory");
}

// grid: clusters of two blocks.
template <bool GATED>
__global__ void __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ Args in, const __grid_constant__ Maps maps) {
    extern __shared__ unsigned char smem_raw[];
    const unsigned raw = smem_u32(smem_raw) & 0xFFFFFFu;  // (within a cluster the block's number is above)
    unsigned char* ring = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
    Shared* sh = reinterpret_cast<Shared*>(ring + RING_BYTES);
    const int warp = warps_own(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int rank = warps_own(cluster_rank());
    const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;

    const int slots = in.slots, slot_bytes = in.slot_bytes;
    if (threadIdx.x == 0) {
        for (int s = 0; s < slots; ++s) {
            mbar_init(&sh->full[s], 1);  // (the first block's, for the copies of both)
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh->acc_full[b], 1);
            mbar_init(&sh->acc_empty[b], 2 * WORKERS);
        }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = warps_own(sh->tmem_base);
    ie_pdl_trigger();
    ie_pdl_wait();

    const int total = min(in.count[0], in.max_tiles) * in.feature_blocks, nkb = in.kbs;
    auto tile_at = [&](int t) {  // (expert, first place, pairs, the tile's number along the features)
        const int r = t / in.feature_blocks;
        int4 v = in.tiles[r];
        v.z = min(v.z, in.most);
        v.w = t - r * in.feature_blocks;
        return v;
    };

    if (warp == 0) {
        const bool one = elect_one();
        int use = 0, s = 0, phase = 0;  // copies so far, over all tiles; their slot, and how often it was used
        bool ok = true;
        for (int t = cluster; t < total && ok; t += clusters) {
            const int4 tile = tile_at(t);
            const int n = warps_own(tile.z), cols = columns(n), rows = cols / 2, bytes = rows * BK * 2;
            const int block = min(2 * warps_own(tile.w) + rank, in.w_blocks - 1);  // (an odd number of them: the last one again, unused)
            int x = (warps_own(tile.y) + rank * rows) >> 3, w = (warps_own(tile.x) * in.w_blocks + block) * nkb * (W_BYTES / 2048);  // (rows of the maps)
            for (int kb = 0; kb < nkb; ++kb, ++use) {
                if (use >= slots && !warp_wait(&sh->empty[s], phase ^ 1)) { ok = false; break; }
                if (one) {
                    unsigned char* at = ring + (size_t)s * slot_bytes;
                    const unsigned bar = in_first(&sh->full[s]);
                    if (rank == 0) mbar_expect_tx(&sh->full[s], 2 * (W_BYTES + parts(n) * bytes));
                    load_pair(at, &maps.w, w, bar);
                    load_rows(at + W_BYTES, maps.x, x, rows >> 3, bar);
                    if (n > MOST_COLS) load_rows(at + W_BYTES + bytes, maps.x, x + (cols >> 3), rows >> 3, bar);
                }
                __syncwarp();
                w += W_BYTES / 2048;
                x += in.places >> 3;
                if (++s == slots) { s = 0; phase ^= 1; }
            }
        }
        if (!ok) sh->failed = 1;
        else
            for (int u = max(use - slots, 0); u < use; ++u) mbar_wait_compact(&sh->empty[u % slots], (u / slots) & 1);  // (none is in flight at the end)
        __syncwarp();
    } else if (warp == 1) {
        const bool one = elect_one();
        int s = 0, phase = 0, turn = 0;
        bool ok = true;
        const unsigned w_low = umma_desc_low(smem_u32(ring));
        for (int t = cluster; rank == 0 && t < total && ok; t += clusters) {
            const int n = warps_own(tile_at(t).z), cols = columns(n);
            const unsigned idesc = umma_idesc_bf16(256, cols), second = (unsigned)(cols / 2 * BK * 2) >> 4;
            for (int part = 0; part < parts(n); ++part) {
                const int use_of = turn + part;
                if (use_of >= 2 && !warp_wait_cluster(&sh->acc_empty[use_of & 1], (use_of / 2 - 1) & 1)) ok = false;
            }
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned acc = tmem + (turn & 1) * MOST_COLS, acc2 = tmem + (~turn & 1) * MOST_COLS;
            for (int kb = 0; kb < nkb; ++kb) {
                if (!warp_wait_cluster(&sh->full[s], phase)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (one) {
                    const unsigned w0 = w_low + s * (slot_bytes >> 4), x0 = w0 + (W_BYTES >> 4);
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks) {  // 32 bytes further along k per step
                        mma<true>(acc, w0 + 2 * ks, x0 + 2 * ks, idesc, kb > 0 || ks > 0);
                        if (n > MOST_COLS) mma<true>(acc2, w0 + 2 * ks, x0 + second + 2 * ks, idesc, kb > 0 || ks > 0);
                    }
                    pair_commit(&sh->empty[s]);
                    if (kb + 1 == nkb)
                        for (int part = 0; part < parts(n); ++part) pair_commit(&sh->acc_full[(turn + part) & 1]);
                }
                __syncwarp();
                if (++s == slots) { s = 0; phase ^= 1; }
            }
            turn += parts(n);
        }
        if (!ok) sh->failed = 1;
        __syncwarp();
    } else {
        const int group = warp & 3, side = (warp - 2) >> 2;  // a warp reads the 32 lanes 32 (warp % 4) ..
        int turn = 0;
        bool ok = true;  // (after a wait that ran out nothing is waited for or read, but the warps still meet at their barriers)
        for (int t = cluster; t < total; t += clusters) {
            const int4 tile = tile_at(t);
            const int cols = columns(tile.z);
            for (int part = 0; part < parts(tile.z); ++part, ++turn) {
                const int first = tile.y + part * cols, n = min(tile.z - part * cols, cols), buf = turn & 1;
                if (!GATED) {
                    const int c = threadIdx.x - 64;
                    if (c < n) {
                        const int pair = in.order[first + c], token = pair / in.top;
                        sh->row_of[buf][c] = (pair - token * in.top) * in.N + token;
                        sh->weight_of[buf][c] = in.weights[pair];
                    }
                    named_barrier(1, WORKERS * 32);
                }
                if (lane == 0 && ok && !mbar_wait_compact(&sh->acc_full[buf], (turn / 2) & 1)) { ok = false; sh->failed = 1; }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) continue;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned acc = tmem + buf * MOST_COLS + ((unsigned)(group * 32) << 16);
                const int row = group * 32 + lane;
                if (GATED) {
                    const int f = (2 * tile.w + rank) * 64 + (row >> 4) * 8 + (row & 7);
                    const int own = f < in.w_blocks * 64 ? n : 0;
                    for (int c0 = side * 16; c0 < cols; c0 += 32) {
                        float a[16];
                        tmem_ld16(a, acc + c0);
                        put_gated(in, a, lane & 8, first + c0, own - c0, f);
                    }
                } else {
                    const int f = (2 * tile.w + rank) * ROWS + row, own = f < in.F ? n : 0;
                    float* out = in.out + f;
                    for (int c0 = side * 16; c0 < cols; c0 += 32) {
                        float a[16];
                        tmem_ld16(a, acc + c0);
#pragma unroll
                        for (int i = 0; i < 16; i += 4) {
                            const int4 row4 = *reinterpret_cast<const int4*>(&sh->row_of[buf][c0 + i]);
                            const float4 w4 = *reinterpret_cast<const float4*>(&sh->weight_of[buf][c0 + i]);
                            const int rows[4] = {row4.x, row4.y, row4.z, row4.w};
                            const float ws[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (c0 + i + j < own) out[(size_t)rows[j] * in.F] = ws[j] * a[i + j];
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive_at(in_first(&sh->acc_empty[buf]));
            }
        }
        __syncwarp();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    if (threadIdx.x == 0 && sh->failed) ie_report(in.err, IE_ERR_TIMEOUT, blockIdx.x, GATED);
    cluster_barrier();
}

constexpr int FEW_PAIRS = 64, FEW_WORKERS = 4, FEW_THREADS = (2 + FEW_WORKERS) * 32, FEW_RING = 72 * 1024, FEW_SLOTS = 4;
// Rows of x are announced when the next ones have been asked for: with three slots a later announcement would have to wait for
// the products that read the slot in between.
constexpr int LAG = 1;
struct __align__(8) FewShared {
    unsigned long long full[FEW_SLOTS], empty[FEW_SLOTS], acc_done;
    unsigned tmem_base;
    int failed;
    int row_of[FEW_PAIRS];  // a pair's row of x, or of the output
    float weight_of[FEW_PAIRS];
};
constexpr size_t FEW_SMEM = (size_t)FEW_RING + sizeof(FewShared) + 1024;

__device__ __forceinline__ void cp16(unsigned dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// grid: (tiles of 128 rows of weights, tiles of pairs)
template <bool GATED>
__global__ void __launch_bounds__(FEW_THREADS, 3)
gemm_few_kernel(const __grid_constant__ Args in) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    FewShared* sh = reinterpret_cast<FewShared*>(ring + FEW_RING);
    const int warp = warps_own(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (GATED) ie_pdl_wait();
    ie_pdl_trigger();
    if ((int)blockIdx.y >= __ldcg(in.count)) {  // (the whole block, before any barrier)
        if (!GATED) ie_pdl_leave();
        return;
    }
    const int4 tile = __ldcg(in.tiles + blockIdx.y);
    const int n = min(warps_own(tile.z), FEW_PAIRS), n_pad = (n + 15) & ~15, x_bytes = n_pad * BK * 2, slot_bytes = W_BYTES + x_bytes;
    const int slots = min(FEW_RING / slot_bytes, FEW_SLOTS);  // at least 3 (a slot is a multiple of 1 KB)
    const int nkb = in.kbs;

    if (threadIdx.x == 0) {
        for (int s = 0; s < slots; ++s) {
            mbar_init(&sh->full[s], GATED ? 1 + FEW_WORKERS : 1);
            mbar_init(&sh->empty[s], 1);
        }
        mbar_init(&sh->acc_done, 1);
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(FEW_PAIRS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x >= 64 && threadIdx.x < 64 + FEW_PAIRS) {
        const int c = threadIdx.x - 64;
        const int pair = c < n ? __ldcg(in.order + tile.y + c) : -1;
        const int token = pair / in.top, choice = pair - token * in.top;
        sh->row_of[c] = pair < 0 ? -1 : GATED ? token : choice * in.N + token;
        if (!GATED) sh->weight_of[c] = pair >= 0 ? __ldcg(in.weights + pair) : 0.f;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = warps_own(sh->tmem_base);

    if (warp == 0) {
        const bool one = elect_one();
        const unsigned char* w = w_tile(in, warps_own(tile.x), blockIdx.x, 0);
        const unsigned char* y = in.x + (size_t)warps_own(tile.y) * BK * 2;
        auto ask_w = [&](int kb, int s) {
            if (!one) return;
            mbar_expect_tx(&sh->full[s], W_BYTES + (GATED ? 0 : x_bytes));
            load_run(ring + (size_t)s * slot_bytes, w + (size_t)kb * W_BYTES, W_BYTES, &sh->full[s]);
        };
        auto ask_y = [&](int kb, int s) {
            if (one) load_run(ring + (size_t)s * slot_bytes + W_BYTES, y + (size_t)kb * in.places * BK * 2, x_bytes, &sh->full[s]);
        };
        const int early = min(slots, nkb);
        for (int kb = 0; kb < early; ++kb) ask_w(kb, kb);
        __syncwarp();
        if (!GATED) {
            ie_pdl_wait();  // (y is the kernel's before)
            for (int kb = 0; kb < early; ++kb) ask_y(kb, kb);
            __syncwarp();
        }
        int s = 0, phase = 0;
        for (int kb = early; kb < nkb; ++kb) {
            if (!warp_wait(&sh->empty[s], phase)) { sh->failed = 1; break; }
            ask_w(kb, s);
            if (!GATED) ask_y(kb, s);
            __syncwarp();
            if (++s == slots) { s = 0; phase ^= 1; }
        }
        __syncwarp();
    } else if (warp == 1) {
        const bool one = elect_one();
        const unsigned idesc = umma_idesc_bf16(ROWS, n_pad), w_low = umma_desc_low(smem_u32(ring));
        bool ok = true;
        int s = 0, phase = 0;
        for (int kb = 0; kb < nkb; ++kb) {
            if (!warp_wait(&sh->full[s], phase)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (one) {
                const unsigned w0 = w_low + s * (slot_bytes >> 4), x0 = w0 + (W_BYTES >> 4);
#pragma unroll
                for (int ks = 0; ks < BK / 16; ++ks) mma<false>(tmem, w0 + 2 * ks, x0 + 2 * ks, idesc, kb > 0 || ks > 0);
                umma_commit(&sh->empty[s]);
            }
            __syncwarp();
            if (++s == slots) { s = 0; phase ^= 1; }
        }
        if (!ok) sh->failed = 1;
        if (one) umma_commit(&sh->acc_done);
        __syncwarp();
    } else {
        const int worker = threadIdx.x - 64;
        if (GATED) {
            // x's rows: eight threads a row, 16 rows at a time
            const int chunk = worker & 7, r0 = worker >> 3;
            const bf16* src[FEW_PAIRS / 16];
            const bf16* x = reinterpret_cast<const bf16*>(in.x);
#pragma unroll
            for (int p = 0; p < FEW_PAIRS / 16; ++p) {
                const int row = sh->row_of[r0 + 16 * p];
                src[p] = row >= 0 ? x + (size_t)row * in.K + chunk * 8 : nullptr;
            }
            const unsigned to = (unsigned)((r0 * 8 + (chunk ^ (r0 & 7))) * 16);  // (r0 + 16 p: the same place in its group of eight rows)
            auto announce = [&](int kb) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->full[kb % slots]);
            };
            bool ok = true;
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % slots;
                if (kb >= slots && !mbar_wait_compact(&sh->empty[s], ((kb / slots) - 1) & 1)) { ok = false; break; }
                const unsigned base = smem_u32(ring + (size_t)s * slot_bytes + W_BYTES) + to;
                const int bytes = kb * BK + chunk * 8 < in.K ? 16 : 0;  // (beyond K: zeros; K is a multiple of 8)
#pragma unroll
                for (int p = 0; p < FEW_PAIRS / 16; ++p)
                    if (src[p] != nullptr) cp16(base + p * 16 * 128, bytes ? src[p] + kb * BK : x, bytes);
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
        } else {
            ie_pdl_wait();
        }
        const bool ok = mbar_wait_compact(&sh->acc_done, 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (__all_sync(0xffffffffu, ok && !sh->failed)) {
            const int group = warp & 3, row = group * 32 + lane;  // a warp reads the 32 lanes 32 (warp % 4) ..
            const unsigned taddr = tmem + ((unsigned)(group * 32) << 16);
            for (int c0 = 0; c0 < n_pad; c0 += 16) {
                float a[16];
                tmem_ld16(a, taddr + c0);
                if (GATED) {
                    put_gated(in, a, lane & 8, tile.y + c0, n - c0, blockIdx.x * 64 + (row >> 4) * 8 + (row & 7));
                } else {
                    const int f = blockIdx.x * ROWS + row;
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (c0 + i < n && f < in.F) in.out[(size_t)sh->row_of[c0 + i] * in.F + f] = sh->weight_of[c0 + i] * a[i];
                }
            }
        }
        if (!ok) sh->failed = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(FEW_PAIRS) : "memory");
    if (threadIdx.x == 0 && sh->failed) ie_report(in.err, IE_ERR_TIMEOUT, blockIdx.x, blockIdx.y);
}

// xs[k block][place][64] = the tokens' rows of the places' pairs, pieces turned as the tensor cores read them, zeros beyond K.  A warp per place.
__global__ void __launch_bounds__(256)
routed_gather_kernel(const uint4* __restrict__ x, uint4* __restrict__ xs, const int* __restrict__ order, const int* __restrict__ meta,
                     int top, int pieces, int kbs, int places) {
    ie_pdl_trigger();
    ie_pdl_wait();
    const int place = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (place >= meta[1]) return;
    const int pair = order[place];
    if (pair < 0) return;
    const uint4* from = x + (size_t)(pair / top) * pieces;
    for (int i = lane; i < kbs * 8; i += 128) {
        uint4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + 32 * k < pieces ? from[i + 32 * k] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int j = i + 32 * k;
            if (j < kbs * 8) xs[((size_t)(j >> 3) * places + place) * 8 + ((j & 7) ^ (place & 7))] = v[k];
        }
    }
}

// Clusters of two that the device runs at one time (an SM without a partner takes none): with one more than those the last would do its
// tiles when all others have done theirs.
template <bool GATED>
int clusters_at_once() {
    static int known[IE_MAX_DEVICES] = {};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= IE_MAX_DEVICES) return ie_sm_count() / 2 - 8;
    if (known[dev] == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * (ie_sm_count() / 2));
        cfg.blockDim = dim3(THREADS);
        cfg.dynamicSmemBytes = SMEM_BYTES;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, gemm_pair_kernel<GATED>, &cfg) != cudaSuccess || clusters < 1) {
            cudaGetLastError();
            clusters = ie_sm_count() / 2 - 8;
        }
        known[dev] = clusters;
    }
    return known[dev];
}

// Memory as rows of `row_bytes` (a multiple of 16, up to 2 KB), boxes of so many.
bool make_row_map(CUtensorMap* map, const void* base, long long rows, int row_bytes, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (fn == nullptr) return false;
    cuuint64_t dims[2] = {(cuuint64_t)row_bytes / 8, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    cuuint32_t box[2] = {(cuuint32_t)row_bytes / 8, (cuuint32_t)box_rows}, elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool GATED>
int launch(const Args& in, int experts, int few, cudaStream_t s) {
    if (few) {
        static IePerDevice allowed;
        cudaError_t e = ie_allow_smem(allowed, gemm_few_kernel<GATED>, FEW_SMEM);
        if (e != cudaSuccess) return (int)e;
        return ie_launch(gemm_few_kernel<GATED>, dim3(in.w_blocks, in.max_tiles), dim3(FEW_THREADS), FEW_SMEM, s, in);
    }
    static IePerDevice allowed;
    cudaError_t e = ie_allow_smem(allowed, gemm_pair_kernel<GATED>, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    const long long most = (long long)in.max_tiles * in.feature_blocks;
    const int pairs = clusters_at_once<GATED>(), clusters = most < pairs ? (int)most : pairs;
    Args args = in;
    const int rows = in.most <= MOST_COLS ? (in.most + 31) / 32 * 16 : MOST_PAIRS / 2;
    args.slot_bytes = W_BYTES + rows * BK * 2;
    args.slots = RING_BYTES / args.slot_bytes < MOST_SLOTS ? RING_BYTES / args.slot_bytes : MOST_SLOTS;
    Maps maps;
    if (!make_row_map(&maps.w, in.w, (long long)experts * in.w_blocks * in.kbs * (W_BYTES / 2048), 2048, W_BYTES / 2048)) return (int)cudaErrorNotSupported;
    for (int i = 0; i < 4; ++i)
        if (!make_row_map(&maps.x[i], in.x, (long long)in.kbs * in.places / 8, 1024, 16 >> i)) return (int)cudaErrorNotSupported;
    return ie_launch_cluster(gemm_pair_kernel<GATED>, dim3(2 * clusters), dim3(THREADS), SMEM_BYTES, s, dim3(2, 1, 1), args, maps);
}
}  // namespace

// Up to so many tokens the kernel for few of them runs.
IE_API int ie_routed_tiled_few() { return FEW_PAIRS; }

// The most pairs of a tile of a step of N tokens, and the multiple at which an expert's places start, for `routed_sort`.  (An expert that no
// token names twice is one tile up to 320 pairs; a multiple of 32, and so of the places' 8.)
IE_API int ie_routed_tiled_most(int N) { return N <= FEW_PAIRS ? FEW_PAIRS : N <= MOST_COLS ? (N + 31) / 32 * 32 : MOST_PAIRS; }
IE_API int ie_routed_tiled_align() { return 8; }

// Places to have room for: every expert's up to 7 more, and what the last tile's copies read beyond its pairs.
IE_API int ie_routed_tiled_places(int pairs, int experts) { return (pairs + 7 * (pairs < experts ? pairs : experts) + MOST_PAIRS + 7) / 8 * 8; }

// Whether there is room for tiles of up to `most` pairs.
static bool fits(int few, int most, int N) { return most > 0 && most <= (few ? FEW_PAIRS : MOST_PAIRS) && (!few || N <= FEW_PAIRS); }

IE_API int ie_routed_tiled_gather(const void* x, void* xs, const int* order, const int* meta, int places, int top, int K, void* stream) {
    if (places <= 0) return 0;
    if (K % 8 || (((uintptr_t)x | (uintptr_t)xs) & 15)) return (int)cudaErrorInvalidValue;
    return ie_launch(routed_gather_kernel, dim3((places + 7) / 8), dim3(256), 0, (cudaStream_t)stream, (const uint4*)x, (uint4*)xs, order, meta,
                     top, K / 8, (K + BK - 1) / BK, places);
}

// most: the pairs of a tile, as `routed_sort` was told.  y: [k blocks of F][places][64].  few: x holds the tokens' rows [N, K]; else what `gather` wrote.  w: [experts][ceil(F / 64)][ceil(K / 64)] tiles.
IE_API int ie_routed_tiled_gate_up(const void* x, const void* w, void* y, const int* order, const int* tiles, const int* count, int max_tiles,
                                   int experts, int few, int most, int top, int N, int places, int K, int F, float limit, int clamp, float alpha, float up_offset,
                                   int* err, void* stream) {
    if (max_tiles <= 0) return 0;
    if (K <= 0 || F <= 0 || K % 8 || F % 8 || ((((uintptr_t)x | (uintptr_t)w | (uintptr_t)y)) & 15) || !fits(few, most, N) || experts <= 0 || places % 8)
        return (int)cudaErrorInvalidValue;
    Args in = {};
    in.w = (const unsigned char*)w;
    in.x = (const unsigned char*)x;
    in.tiles = (const int4*)tiles;
    in.count = count;
    in.max_tiles = max_tiles;
    in.w_blocks = (F + 63) / 64;
    in.feature_blocks = (in.w_blocks + 1) / 2;
    in.places = places;
    in.kbs = (K + BK - 1) / BK;
    in.K = K;
    in.F = F;
    in.y = (bf16*)y;
    in.order = order;
    in.top = top;
    in.N = N;
    in.most = most;
    in.limit = limit;
    in.clamp = clamp;
    in.alpha = alpha;
    in.up_offset = up_offset;
    in.err = err;
    return launch<true>(in, experts, few, (cudaStream_t)stream);
}

// w: [experts][ceil(H / 128)][ceil(F / 64)] tiles; out: [top, N, H] 32-bit.  few: launched right behind ie_routed_tiled_gate_up.
IE_API int ie_routed_tiled_down(const void* y, const void* w, float* out, const float* weights, const int* order, const int* tiles,
                                const int* count, int max_tiles, int experts, int few, int most, int top, int N, int places, int F, int H, int* err, void* stream) {
    if (max_tiles <= 0) return 0;
    if (H <= 0 || F <= 0 || H % 8 || F % 8 || ((((uintptr_t)y | (uintptr_t)w)) & 15) || !fits(few, most, N) || experts <= 0 || places % 8) return (int)cudaErrorInvalidValue;
    Args in = {};
    in.w = (const unsigned char*)w;
    in.x = (const unsigned char*)y;
    in.tiles = (const int4*)tiles;
    in.count = count;
    in.max_tiles = max_tiles;
    in.w_blocks = (H + ROWS - 1) / ROWS;
    in.feature_blocks = (in.w_blocks + 1) / 2;
    in.places = places;
    in.kbs = (F + BK - 1) / BK;
    in.K = F;
    in.F = H;
    in.out = out;
    in.order = order;
    in.weights = weights;
    in.top = top;
    in.N = N;
    in.most = most;
    in.err = err;
    return launch<false>(in, experts, few, (cudaStream_t)stream);
}
