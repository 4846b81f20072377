// Attention over a paged cache of latent rows [c (RANK) | rotated key part (rot)] on the tcgen05 tensor cores, bfloat16, compiled
// per latent size (-DRANK=N, a multiple of 128 up to 512).  All heads of a token read the same rows, so a tile's query rows are
// (token, head) pairs of one request.
//
// What decides the shape: the outputs of a row are RANK 32-bit numbers, and tensor memory holds 512 columns for 128 lanes, so 128
// rows with 512 outputs each leave no room for their scores.  A PAIR of blocks (a cluster of two, tcgen05 with .cta_group::2 and
// M = 128) therefore serves 128 rows, 64 per block: such an instruction keeps a block's 64 rows in lanes 0..63 with the first
// half of its N columns and in lanes 64..127 with the second half, so that a row's 512 outputs take 256 columns and the scores of
// two key tiles find room beside them.  Each block fetches half of the key rows for S = Q K^T (N is split over the pair) and
// half of the value columns for O += P V; V is the first RANK values of the same rows, read as an MN-major operand as it lies
// in the cache.  Per key tile of 128 and block:
//
//   warps 0..3  softmax: a thread owns half of a row's keys (lanes 0..63: the tile's first 64, lanes 64..127: the others), the two
//               threads of a row tell each other their maxima; P goes to shared memory (the A operand of O += P V).  The outputs
//               are rescaled only when a row's maximum has grown by more than 2^8 or its weight asks for it.
//   warp 4      of the first block issues the pair's instructions: S(0) S(1) | O(0) S(2) | O(1) S(3) | ...
//   warps 5..8  TMA, page by page through the block table, 64 columns x 64 keys at a time, into a ring of 16 KB stages, in turn; the
//               barrier of a stage lives in the first block and counts both blocks' bytes.  The keys run two tiles ahead of the
//               values.  Value rows behind the request's last token (stale memory may hold NaN) are written by hand, as zeros.
//               (A load takes its warp some 100 cycles to issue, and pages of 16 tokens are 68 loads a tile: one warp alone needed
//               7,800 cycles a tile, the matrix instructions 3,700.)
//
// Measured (a 2,000-token prompt, 16 heads on rows of 512 + 64, pages of 16): about 129 us, against 454 us of the warp-level kernel, whose time
// went into the fragments that every warp re-read from shared memory.  A key tile takes some 6,200 cycles (5,900 while the reference only
// moved by 2^8): 36 instructions of 33 cycles and
// 16 of 65 are 2,200 of them, waits for loads 1,900: the ring covers 1,800 cycles, about what a load needs from L2 to its barrier.
//
// Every wait is bounded; one that gives up sets the error flag (llme_latent_pair_status()) and the block drains and returns.
#include <cuda.h>

#include "common.cuh"
#include "kernel_args.h"

#ifndef RANK
#error "compile with -DRANK=<latent size>"
#endif
static_assert(RANK % 128 == 0 && RANK >= 128 && RANK <= 512, "RANK must be a multiple of 128 up to 512");

LLME_API const char* llme_last_error() { return llme_error_buffer(); }

namespace {
#include "umma.cuh"

constexpr int PAIR_ROWS = 128, ROWS = 64;         // (token, head) rows of a pair, of a block
constexpr int BN = 128;                           // keys per tile
constexpr int CHUNK = 8192;                       // 64 rows of 64 values: 128-byte rows with the 128-byte swizzle
constexpr int STAGE = 2 * CHUNK;
constexpr int VC = RANK / 128;                    // 64-column chunks of a block's half of the value columns
constexpr int VG = (VC + 1) / 2;                  // stages per 64 keys of them
constexpr int MAX_STAGES = 8;
constexpr int LOADERS = 4;                         // warps that issue the loads
constexpr int BLOCK = 32 * (4 + 1 + LOADERS);
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE = 8.0f;

struct Args {
    const bf16* cache; bf16* out;
    const float* sink;
    const int* rows; const int* cu_q_lens; const int* ctx_lens; const int* table_rows; const int* block_tables;
    int max_blocks, nh, width, page_size, stages;
    float scale;
    int window;
};

struct Barriers {
    unsigned long long q_full, full[MAX_STAGES], empty[MAX_STAGES], s_full[2], p_full[2], pv_done;
    unsigned tmem_base;
    int abort_flag;
    float row_max[2][2][ROWS];     // [tile parity][half of the keys][row]
    float row_l[2][2][ROWS];       // likewise: the sums before the tile
    float row_sum[2][ROWS];
};

// mbar_wait() for a barrier on which threads of the other block arrive behind writes of their own
__device__ __forceinline__ bool wait_cluster(unsigned long long* bar, unsigned parity, volatile int* abort_flag, int where) {
    for (unsigned i = 0; i < WAIT_LIMIT; ++i) {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if ((i & 1023u) == 1023u && *abort_flag) return false;
    }
    *abort_flag = where;
    atomicCAS(&g_status, 0, where);
    return false;
}
// arms a barrier (of either block) for bytes that TMA loads will bring; orders nothing by itself: writes that the waiting block is to
// see need a fence of cluster scope in front
__device__ __forceinline__ void arrive_expect_cluster(unsigned cluster_addr, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr), "r"(bytes) : "memory");
}
// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// MN-major operand (value rows as they lie in the cache): 64-column chunks CHUNK bytes apart, groups of eight keys 1024 bytes apart
__device__ __forceinline__ unsigned long long desc_mn(const void* tile) {
    unsigned long long d = umma_desc(tile) & ~((unsigned long long)0x3FFF << 16);
    return d | (unsigned long long)(CHUNK >> 4) << 16;
}
__host__ __device__ constexpr unsigned idesc_pv(int N) { return umma_idesc(PAIR_ROWS, N) | (1u << 16); }
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_st_32x32(unsigned addr, const unsigned (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
__device__ __forceinline__ unsigned pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<unsigned*>(&h);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(BLOCK, 1)
latent_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_c, Args a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int KC = (a.width + 63) >> 6;                         // 64-column chunks of a row
    const int KG = (KC + 1) >> 1;                               // stages of a block's half of a key tile
    unsigned char* q_s = smem;                                  // [KC][64 rows][128 B]
    unsigned char* p_s = q_s + KC * CHUNK;                      // [2][2 halves of the keys][64 rows][128 B]
    unsigned char* ring = p_s + 2 * STAGE;
    Barriers* bar = reinterpret_cast<Barriers*>(ring + a.stages * STAGE);
    volatile int* abort_flag = &bar->abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const int r = a.rows[blockIdx.y], H = a.nh;
    const int tok0 = a.cu_q_lens[r], q_len = a.cu_q_lens[r + 1] - tok0;
    const int n_rows = q_len * H;
    // the last rows of a prompt see the most keys: their blocks are launched first
    const int row0 = ((int)(gridDim.x >> 1) - 1 - (int)(blockIdx.x >> 1)) * PAIR_ROWS;
    if (row0 >= n_rows) return;                                 // (both blocks of the pair)
    const int ctx = a.ctx_lens[r], first_pos = ctx - q_len;
    const int hi_max = first_pos + (min(row0 + PAIR_ROWS, n_rows) - 1) / H;                        // the farthest key any row sees
    const int lo_min = a.window > 0 ? max(0, first_pos + row0 / H - a.window + 1) : 0;             // the nearest
    const int tile_first = lo_min / BN, n_tiles = hi_max / BN + 1 - tile_first;
    const int* bt = a.block_tables + (size_t)a.table_rows[r] * a.max_blocks;

    if (threadIdx.x == 0) {
        mbar_init(&bar->q_full, 2);
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(&bar->full[s], 2);                        // both blocks' loads
            mbar_init(&bar->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bar->s_full[b], 1);
            mbar_init(&bar->p_full[b], 8);                      // the softmax warps of both blocks
        }
        mbar_init(&bar->pv_done, 1);
        bar->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bar->tmem_base)), "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = bar->tmem_base;
    const unsigned tmem_o = tmem, tmem_s = tmem + RANK / 2;     // outputs; scores of two key tiles, 64 columns each

    if (warp > 4) {
        // ------------------------------------------------------------------ loads: the stages are dealt out to the warps in turn
        if (warp == 5 && lane == 0) {
            const unsigned qbar = map_to_cta(smem_u32(&bar->q_full), 0);
            arrive_expect_cluster(qbar, (unsigned)(KC * CHUNK));
            for (int c = 0; c < KC; ++c) tma_load_2d_pair(q_s + c * CHUNK, &map_q, c * 64, tok0 * H + row0 + (int)rank * ROWS, qbar);
        }
        __syncwarp();
        const int ps = a.page_size, bs = ps < 64 ? ps : 64;     // rows of one load
        const int bs_shift = __ffs(bs) - 1, nb_shift = 6 - bs_shift, nb = 1 << nb_shift;
        // The page that holds box `lane` of a tile, or -1: it lies behind the request's last token, or before every key that is
        // seen (its page may be gone); and the place in the page where the box begins.
        struct Box { int page, off; };
        auto box_of = [&](int i) -> Box {
            const int j = (tile_first + i) * BN + (lane << bs_shift);
            if (i >= n_tiles || lane >= 2 * nb || j >= ctx || j + bs - 1 < lo_min) return {-1, 0};
            const int blk = j / ps;
            return {bt[blk], j - blk * ps};
        };
        unsigned s = 0, phase = 1;
        int turn = warp - 5;                                    // stages until this warp's next one
        bool ok = true;
        // One stage: `n_chunks` 64-column chunks from column x0 on, of the 64 keys of half `kh` of tile i.
        auto load_stage = [&](int i, int kh, int x0, int n_chunks, Box tile_box, bool values) {
            if (!ok) return;
            const unsigned at_s = s, at_phase = phase;
            if (++s == (unsigned)a.stages) { s = 0; phase ^= 1u; }
            if (turn-- != 0) return;
            turn = LOADERS - 1;
            ok = mbar_wait(&bar->empty[at_s], at_phase, abort_flag, 1) && !*abort_flag;
            ok = __all_sync(0xffffffffu, ok);                   // (a lane that gave up takes the others with it: what follows needs them all)
            if (!ok) return;
            unsigned char* stage = ring + at_s * STAGE;
            const int cc = lane >> nb_shift, box = lane & (nb - 1);
            const int j_half = (tile_first + i) * BN + kh * 64, j = j_half + (box << bs_shift);
            const int page = __shfl_sync(0xffffffffu, tile_box.page, (kh << nb_shift) + box);
            const int row = page * ps + __shfl_sync(0xffffffffu, tile_box.off, (kh << nb_shift) + box);
            const bool mine = cc < n_chunks;
            // Key rows that no query of the tile sees give scores that are masked.  Value rows must be finite: what lies behind the
            // request's last token may be anything, what lies between the tile's last key and that is finite.
            const bool whole = mine && page >= 0 && (!values || j + bs <= ctx);
            const unsigned whole_mask = __ballot_sync(0xffffffffu, whole);
            const unsigned hand = values ? __ballot_sync(0xffffffffu, mine && !whole) : 0u;
            if (hand) {
                for (unsigned rest = hand; rest; rest &= rest - 1) {
                    const int src = __ffs(rest) - 1;
                    const int b_row = (src & (nb - 1)) << bs_shift, chunk = src >> nb_shift;
                    const int from = __shfl_sync(0xffffffffu, page >= 0 ? row : -1, src);
#pragma unroll 4
                    for (int e = lane; e < bs * 8; e += 32) {
                        const int rr = e >> 3, q = e & 7, at = b_row + rr;
                        uint4 v = make_uint4(0u, 0u, 0u, 0u);
                        if (from >= 0 && j_half + at < ctx)
                            v = *reinterpret_cast<const uint4*>(a.cache + (size_t)(from + rr) * a.width + x0 + chunk * 64 + q * 8);
                        *reinterpret_cast<uint4*>(stage + chunk * CHUNK + at * 128 + ((q ^ (at & 7)) << 4)) = v;
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            __syncwarp();
            const unsigned full = map_to_cta(smem_u32(&bar->full[at_s]), 0);
            if (lane == 0) {
                // rows written by hand: the warp's writes, which this lane knows of from __syncwarp(), come before its arrival for
                // the block that waits (a fence in front of __syncwarp() would order this lane's own only)
                if (hand) asm volatile("fence.acq_rel.cluster;" ::: "memory");
                arrive_expect_cluster(full, (unsigned)__popc(whole_mask) * (unsigned)(bs * 128));
            }
            __syncwarp();
            if (whole) tma_load_2d_pair(stage + cc * CHUNK + (box << bs_shift) * 128, &map_c, x0 + cc * 64, row, full);
        };
        auto load_keys = [&](int i, Box tile_box) {
            for (int g = 0; g < KG; ++g) load_stage(i, (int)rank, g * 128, min(2, KC - 2 * g), tile_box, false);
        };
        Box box_0 = box_of(0), box_1 = box_of(1), box_2 = box_of(2);
        load_keys(0, box_0);
        if (n_tiles > 1) load_keys(1, box_1);
        for (int i = 0; i < n_tiles && ok; ++i) {
            const Box box_3 = box_of(i + 3);
            for (int kh = 0; kh < 2; ++kh)
                for (int g = 0; g < VG; ++g) load_stage(i, kh, (int)rank * (RANK / 2) + g * 128, min(2, VC - 2 * g), box_0, true);
            if (i + 2 < n_tiles) load_keys(i + 2, box_2);
            box_0 = box_1;
            box_1 = box_2;
            box_2 = box_3;
        }
        if (*abort_flag) {
            for (int i = 0; i < 200; ++i) __nanosleep(5000);    // gave up: copies still in flight land before the block exits
        }
    } else if (warp == 4) {
        // ------------------------------------------------------------------ matrix instructions
        // The whole warp walks the loop and one elected lane issues: the operands' descriptors then stay in uniform registers.  (Behind a
        // branch on the lane an instruction takes 52 cycles to issue, so 23 to 30: M = 128, N = 128 needs 33 of the pipe, N = 256 65.)
        if (rank == 0) {
            constexpr unsigned id_s = umma_idesc(PAIR_ROWS, BN);
            const unsigned long long dq = umma_desc(q_s), dp = umma_desc(p_s), dk = umma_desc(ring), dv = desc_mn(ring);
            const unsigned d_o = __shfl_sync(0xffffffffu, tmem_o, 0), d_s = __shfl_sync(0xffffffffu, tmem_s, 0);
            unsigned s = 0, phase = 0;
            bool ok = __all_sync(0xffffffffu, mbar_wait(&bar->q_full, 0, abort_flag, 20));
            auto next_stage = [&](bool hand) {
                ok = ok && (hand ? wait_cluster(&bar->full[s], phase, abort_flag, 21) : mbar_wait(&bar->full[s], phase, abort_flag, 21));
                ok = __all_sync(0xffffffffu, ok);
                if (ok) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            };
            auto free_stage = [&]() {
                if (elect_one()) umma_commit_pair(&bar->empty[s]);
                __syncwarp();
                if (++s == (unsigned)a.stages) { s = 0; phase ^= 1u; }
            };
            auto issue_s = [&](int i) {
                const unsigned d = d_s + (unsigned)((i & 1) * 64);
                for (int g = 0; g < KG; ++g) {
                    next_stage(false);
                    if (!ok) return;
                    const int n = min(2, KC - 2 * g);
                    const unsigned long long da = dq + (unsigned long long)(2 * g * (CHUNK >> 4)), db = dk + s * (STAGE >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) umma_bf16_pair(d, da + 2 * k, db + 2 * k, id_s, (g | k) ? 1u : 0u);
                        if (n == 2) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) umma_bf16_pair(d, da + (CHUNK >> 4) + 2 * k, db + (CHUNK >> 4) + 2 * k, id_s, 1u);
                        }
                    }
                    __syncwarp();
                    free_stage();
                }
                if (elect_one()) umma_commit_pair(&bar->s_full[i & 1]);
                __syncwarp();
            };
            auto issue_pv = [&](int i) {
                ok = __all_sync(0xffffffffu, ok && wait_cluster(&bar->p_full[i & 1], (unsigned)(i >> 1) & 1u, abort_flag, 22));
                const bool hand = (tile_first + i) * BN + BN > ctx || (tile_first + i) * BN < lo_min;      // value rows written by hand among them
                for (int kh = 0; kh < 2; ++kh) {
                    const unsigned long long da = dp + (unsigned long long)((i & 1) * (STAGE >> 4) + kh * (CHUNK >> 4));
#pragma unroll
                    for (int g = 0; g < VG; ++g) {
                        next_stage(hand);
                        if (!ok) return;
                        const unsigned long long db = dv + s * (STAGE >> 4);
                        constexpr unsigned id_2 = idesc_pv(256), id_1 = idesc_pv(128);
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < 4; ++k)                                // 16 keys: two groups of eight, 2,048 bytes
                                umma_bf16_pair(d_o + (unsigned)(g * 128), da + 2 * k, db + 128 * k, VC - 2 * g >= 2 ? id_2 : id_1, (i | kh | k) ? 1u : 0u);
                        }
                        __syncwarp();
                        free_stage();
                    }
                }
                if (elect_one()) umma_commit_pair(&bar->pv_done);
                __syncwarp();
            };
            if (ok) issue_s(0);
            if (ok && n_tiles > 1) issue_s(1);
            for (int i = 0; i < n_tiles && ok; ++i) {
                issue_pv(i);
                if (ok && i + 2 < n_tiles) issue_s(i + 2);
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax and output
        const int quarter = warp, kh = quarter >> 1;        // lanes 32 quarter ..: 32 rows, one half of the keys (and of the output columns)
        const int row = (quarter & 1) * 32 + lane;
        const int g_row = row0 + (int)rank * ROWS + row;
        const bool row_ok = g_row < n_rows;
        const int p = row_ok ? first_pos + g_row / H : -1;
        const int plo = a.window > 0 ? max(0, p - a.window + 1) : 0;
        const unsigned lane_off = (unsigned)(quarter * 32) << 16;
        const float sc = a.scale * LOG2E;
        const unsigned p_bar = map_to_cta(smem_u32(&bar->p_full[0]), 0);
        auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + (quarter & 1)) : "memory"); };
        // what every row of this warp sees entirely, without a mask
        const int w_first = row0 + (int)rank * ROWS + (quarter & 1) * 32;
        const int see_hi = w_first + 31 < n_rows ? first_pos + w_first / H : -1;
        const int see_lo = a.window > 0 ? max(0, first_pos + (w_first + 31) / H - a.window + 1) : 0;
        const bool with_sink = a.sink != nullptr && row_ok;
        float m_ref = with_sink ? a.sink[g_row % H] * LOG2E : -INFINITY;
        float l_run = with_sink && kh == 0 ? 1.0f : 0.0f;       // the sink counts once
        bool unseen = true;                                     // no key of the row so far
        bool ok = true;
        for (int i = 0; i < n_tiles; ++i) {
            const int b = i & 1, j0 = (tile_first + i) * BN + kh * 64;
            ok = ok && mbar_wait(&bar->s_full[b], (unsigned)(i >> 1) & 1u, abort_flag, 30);
            ok = __all_sync(0xffffffffu, ok);                   // (what follows needs the whole warp)
            unsigned v[2][32];
            float own = -INFINITY;
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tmem_ld_32x32(tmem_s + lane_off + (unsigned)(b * 64), v[0]);
                tmem_ld_32x32(tmem_s + lane_off + (unsigned)(b * 64 + 32), v[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (!(j0 >= see_lo && j0 + 63 <= see_hi)) {
#pragma unroll
                    for (int e = 0; e < 64; ++e) {
                        const int j = j0 + e;
                        if (j > p || j < plo) v[e >> 5][e & 31] = 0xff800000u;
                    }
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int e = 0; e < 64; ++e) mx[e & 3] = fmaxf(mx[e & 3], __uint_as_float(v[e >> 5][e & 31]));
                own = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            }
            // (both threads of a row come here once per tile, also after a wait has given up)
            bar->row_max[b][kh][row] = own;
            bar->row_l[b][kh][row] = l_run;
            pair_sync();
            if (!ok) continue;
            const float m_true = fmaxf(own, bar->row_max[b][kh ^ 1][row]) * sc;
            // Relative to the row's true maximum the largest probability is one, which bfloat16 holds exactly; relative to an older
            // reference, or to the sink, it is rounded like the others.  It is kept exact where it weighs: in the first tile that the
            // row sees, and where it is more than a 64th of the row's sum.  Error of the layer, a 2,000-token prompt (the warp-level
            // kernel: 4.2194e-3): 4.2285e-3 with neither this nor the rounded probabilities' sum, 4.2215e-3 with the latter, 4.2183e-3 with both.
            const bool move = m_true > m_ref + RESCALE || (m_true > m_ref && (unseen || fast_exp2(m_true - m_ref) * 64.0f > l_run + bar->row_l[b][kh ^ 1][row]));
            unseen = unseen && m_true == -INFINITY;
            if (__any_sync(0xffffffffu, move)) {
                const float m_new = move ? m_true : m_ref;
                const float corr = move ? fast_exp2(m_ref - m_new) : 1.0f;      // (exp2 of -inf: 0, nothing had been seen)
                l_run *= corr;
                m_ref = m_new;
                if (i > 0) {
                    // at rest once O(i - 1) has been added; O(i) waits for this warp's probabilities
                    ok = __all_sync(0xffffffffu, mbar_wait(&bar->pv_done, (unsigned)(i - 1) & 1u, abort_flag, 31));
                    if (ok) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                        for (int c = 0; c < RANK / 2; c += 32) {
                            unsigned o[32];
                            tmem_ld_32x32(tmem_o + lane_off + (unsigned)c, o);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
                            tmem_st_32x32(tmem_o + lane_off + (unsigned)c, o);
                        }
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    }
                }
            }
            if (!ok) continue;
            const float ref = m_ref == -INFINITY ? 0.0f : m_ref;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            unsigned char* p_row = p_s + b * STAGE + kh * CHUNK + row * 128;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                uint4 pk;
                unsigned* pw = reinterpret_cast<unsigned*>(&pk);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int at = q * 8 + 2 * e;
                    const float e0 = fast_exp2(fmaf(__uint_as_float(v[at >> 5][at & 31]), sc, -ref));          // a masked score is -inf: exactly 0
                    const float e1 = fast_exp2(fmaf(__uint_as_float(v[at >> 5][(at & 31) + 1]), sc, -ref));
                    const __nv_bfloat162 h = __floats2bfloat162_rn(e0, e1);
                    const float2 rounded = __bfloat1622float2(h);        // the sum of what is multiplied with the values
                    sum[e] += rounded.x + rounded.y;
                    pw[e] = *reinterpret_cast<const unsigned*>(&h);
                }
                *reinterpret_cast<uint4*>(p_row + ((q ^ (row & 7)) << 4)) = pk;
            }
            l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(p_bar + (unsigned)(b * 8));
        }
        // S(n - 1) was issued behind O(n - 3): the last two are waited for one after the other (a parity tells neighbours apart only)
        if (n_tiles > 1) ok = ok && mbar_wait(&bar->pv_done, (unsigned)(n_tiles - 2) & 1u, abort_flag, 32);
        ok = ok && mbar_wait(&bar->pv_done, (unsigned)(n_tiles - 1) & 1u, abort_flag, 32) && !*abort_flag;
        ok = __all_sync(0xffffffffu, ok);
        bar->row_sum[kh][row] = l_run;
        pair_sync();
        l_run += bar->row_sum[kh ^ 1][row];
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
            // 32 rows x 64 columns at a time through shared memory (the queries' place, which nothing reads any more), so that a
            // store writes whole 128-byte pieces of rows
            unsigned char* stage = q_s + warp * 4096;
#pragma unroll 1
            for (int c = 0; c < RANK / 2; c += 64) {
                unsigned o[2][32];
                tmem_ld_32x32(tmem_o + lane_off + (unsigned)c, o[0]);
                tmem_ld_32x32(tmem_o + lane_off + (unsigned)(c + 32), o[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    uint4 pk;
                    unsigned* pw = reinterpret_cast<unsigned*>(&pk);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int at = q * 8 + 2 * e;
                        pw[e] = pack2(__uint_as_float(o[at >> 5][at & 31]) * inv, __uint_as_float(o[at >> 5][(at & 31) + 1]) * inv);
                    }
                    *reinterpret_cast<uint4*>(stage + lane * 128 + ((q ^ (lane & 7)) << 4)) = pk;
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int rr = k * 4 + (lane >> 3), q = lane & 7;
                    if (w_first + rr < n_rows)
                        *reinterpret_cast<uint4*>(a.out + ((size_t)tok0 * H + w_first + rr) * RANK + kh * (RANK / 2) + c + q * 8) =
                            *reinterpret_cast<const uint4*>(stage + rr * 128 + ((q ^ (rr & 7)) << 4));
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                       // a pair leaves together
    if (warp == 4) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
    }
}

size_t smem_bytes(int chunks, int stages) { return 1024 + (size_t)chunks * CHUNK + 2 * STAGE + (size_t)stages * STAGE + sizeof(Barriers); }

int stages_for(int chunks) {
    int s = MAX_STAGES;
    while (s > 0 && smem_bytes(chunks, s) > 232448) --s;
    return s;
}

}  // namespace

// Whether the kernel takes rows of RANK + rot values in pages of page_size tokens: rows of whole 16-byte pieces that leave room for four
// stages, pages of 8, 16, 32 or a multiple of 64 tokens.
LLME_API int llme_latent_pair_supports(int rot, int page_size) {
    if (rot < 0 || (RANK + rot) % 8 || stages_for((RANK + rot + 63) / 64) < 4) return 0;
    return page_size == 8 || page_size == 16 || page_size == 32 || (page_size > 0 && page_size % 64 == 0);
}

// 0 if no bounded wait has given up since the last call (synchronises the device).
LLME_API int llme_latent_pair_status() { LLME_TAKE_STATUS(g_status); }

// Requests `rows` of the step, each with any number of new tokens up to `max_q_len`; q has q_rows rows of RANK + rot values in all, the cache
// cache_rows.
LLME_API int llme_latent_pair(const LlmeFastAttnArgs* f, long long q_rows, long long cache_rows, const float* sink, int rot, int max_q_len, cudaStream_t stream) {
    if (f->n_rows <= 0 || max_q_len <= 0) return 0;
    if (!f->q || !f->cache || !f->out || !f->rows || !f->cu_q_lens || !f->ctx_lens || !f->table_rows || !f->block_tables)
        LLME_REFUSE("latent attention: null pointer");
    if (!llme_latent_pair_supports(rot, f->page_size)) LLME_REFUSE("latent attention: rows of %d + %d values in pages of %d do not fit this kernel", RANK, rot, f->page_size);
    if (f->n_rows > 65535 || f->nh < 1) LLME_REFUSE("latent attention: too many requests for one launch");
    if (((uintptr_t)f->q | (uintptr_t)f->cache | (uintptr_t)f->out) % 16) LLME_REFUSE("latent attention: operands must be 16-byte aligned");
    const int width = RANK + rot, chunks = (width + 63) / 64, bs = f->page_size < 64 ? f->page_size : 64;
    alignas(64) CUtensorMap mq, mc;
    if (int rc = make_map(&mq, f->q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q_rows, width, width, ROWS, 64)) return rc;
    if (int rc = make_map(&mc, f->cache, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, cache_rows, width, width, bs, 64)) return rc;
    Args a = {(const bf16*)f->cache, (bf16*)f->out, sink, f->rows, f->cu_q_lens, f->ctx_lens, f->table_rows, f->block_tables,
              f->max_blocks, f->nh, width, f->page_size, stages_for(chunks), f->scale, f->window};
    const size_t smem = smem_bytes(chunks, a.stages);
    static LlmeGrants grants;
    if (cudaError_t e = llme_grant_smem(grants, latent_pair_kernel, smem)) LLME_REFUSE("latent attention: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    const long long pairs = ((long long)max_q_len * f->nh + PAIR_ROWS - 1) / PAIR_ROWS;
    if (pairs > (1 << 29)) LLME_REFUSE("latent attention: too many rows for one launch");
    latent_pair_kernel<<<dim3((unsigned)(2 * pairs), f->n_rows), BLOCK, smem, stream>>>(mq, mc, a);
    LLME_LAUNCH_STATUS();
}
