// The 32-bit product on the tensor cores: both operands as sums of three bfloat16 pieces, six products of pieces each (split32.cuh).
// Included by gemm_f32.cu inside its unnamed namespace; float weights whose rows begin on 16 bytes.
//
// A block takes 128 weight rows (the lanes of tensor memory) and NT rows of A, and walks one segment of K, 64 values at a time:
//   * one warp asks for the weights (TMA, 128-byte swizzle), as soon as the instructions of the chunk that lay there are done;
//   * eight warps split the weights, half a row a thread, and leave the pieces in TENSOR memory, from where the instructions take their
//     first operand: through shared memory the pieces would cost 18 of 26 bytes of traffic a value;
//   * X_WARPS warps split the rows of A, read straight from memory a chunk ahead, and leave their pieces in shared memory as swizzled tiles;
//   * one warp issues 24 instructions a chunk (128 x NT x 16), the small products first;
//   * SUM_WARPS warps read the chunk's sums out of tensor memory and add them in registers: no accumulator is longer than 64 values, for the
//     tensor cores cut off what they add instead of rounding it.
// Three chunks' pieces and two accumulators are in flight.  A wait for a barrier costs 100 to 140 cycles even where the barrier is complete (measured
// alone), so the issuing warp has one a chunk, on which all of its operands and the freed accumulator are counted.
// The segments of K (by K and N alone) are a cluster's blocks: each leaves its sums in shared memory and adds a share of the outputs over
// the blocks in their order.  So an output's additions depend on K and N alone, and a row's bits on no other row.
//
// Infinities, NaN and values that overflow bfloat16 come out of the split as no number; an output that is none is formed again, from its rows
// and in 64 bits, by the warp that stores it.
//
// Rows x outputs x values, us, weights from memory, with the multiply-adds before: 1 / 8 / 32 / 64 / 300 rows of 11008 x 2048 21.9 / 22.0 / 25.0 / 36.9 / 95.5
// (20.1 / 29 / 71 / 120 / 374), of 2048 x 5504 15.1 / 15.6 / 17.2 / 24.3 / 62.6 (17.8 / 24 / 48 / 76 / 201); 300 x 11008 x 2048 is 142 TFLOP/s (850 of bfloat16).  One
// row of 11,008 outputs is the one slower case found: 86 blocks for 148 SMs.  1, 4 and 16 rows of 512 to 4,096 values on 64 to 4,096 outputs are 1.1 to
// 3 times faster than the multiply-adds, so MIN_K and MIN_N need not be larger (64 x 512: 6.6 us, 7.2 to 11.8).  Error against 64 bits, 2-norm
// relative, 601 rows: 1.3e-7 and 1.2e-7 (5.7e-7 and 6.0e-7); what the tensor cores cut off has a sign, but no sum there is longer than 64 values.
// Few rows are bound by the eight warps that split the weights (about 1,000 cycles a chunk, 460 of them waits and barriers), many rows by the
// instructions (1,340 cycles a chunk at 112 rows) and, where all SMs are at work, by what they bring from L2 (60 KB a chunk).  Tried: the sums
// of x's and w's two tf32 parts (three products; error 3.7e-7, same times), pairs of SMs (1.2 times slower: an arrival at the partner's
// barrier takes 425 cycles, one at the block's own 100), mma.sync with a few rows (the same bits; one row of 2048 x 2048 26 us, 7.4 here: its chain of 24).
// All waits are bounded; llme_gemm_f32_status() tells of one that gave up.
#pragma once

namespace split {

#include "umma.cuh"
#include "split32.cuh"

constexpr int CHUNK = 64, W_HALF = BM * 32 * 4, W_CHUNK = 2 * W_HALF, MOST_STAGES = 4, A_COLS = PIECES * CHUNK / 2;      // tensor memory columns of a chunk's weights
constexpr int MIN_K = 512, MIN_N = 64;

struct Args {
    const float* A; const float* W; float* C;
    int M, N, K, segments, segment_chunks, nt, vec_c;
    long long lda, ldw, ldc;
};

struct Barriers {
    unsigned long long w_full[MOST_STAGES];                            // raw weights of a chunk
    unsigned long long ready[MOST_STAGES], done[MOST_STAGES];          // its pieces are there and its accumulator is free; its instructions have finished
    unsigned tmem_base;
    int abort_flag;
};

// SMALL: a few rows of A, whose instructions are short: the warps that split A's rows take the chunks in turn, for what they read is late.
template <bool SMALL> struct Shape {
    static constexpr int MAXN = SMALL ? 32 : 112, STAGES = SMALL ? 4 : 3, W_WARPS = 8, X_SETS = SMALL ? 2 : 1, X_EACH = SMALL ? 2 : 8, SUM_WARPS = SMALL ? 4 : 8;
    static constexpr int X_WARPS = X_SETS * X_EACH, FIRST_SUM = W_WARPS + X_WARPS, ISSUER = FIRST_SUM + SUM_WARPS, THREADS = (ISSUER + 2) * 32;
    static constexpr int COLS = MAXN / (SUM_WARPS / 4);                // columns of sums that a thread holds (at most)
    static constexpr int X_ROWS = X_EACH * 4, X_PIECES = (MAXN + X_ROWS - 1) / X_ROWS;         // rows split at a time; groups of eight values a thread splits
    static_assert(STAGES * A_COLS + 2 * MAXN <= 512 && COLS % 8 == 0, "sizes");
};

// A request to bring a box into L2: it holds nothing back and may come ahead of what is written there.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}

// Outputs that the split does not reach, taken again by a whole warp from rows that begin on 16 bytes: whether a row holds a NaN (then nothing
// else counts), and one output in 64 bits, whose rounding is infinite where the sum is too large and only there.
__device__ __noinline__ bool row_has_nan(const float* __restrict__ x, int K) {
    bool nan = false;
#pragma unroll 4
    for (int k = 4 * ((int)threadIdx.x & 31); k < K; k += 128) {
        const float4 v = row_piece(x, k, K, true);
        nan |= isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w);
    }
    return __any_sync(0xffffffffu, nan);
}
__device__ __noinline__ float plain_dot(const float* __restrict__ x, const float* __restrict__ w, int K) {
    double s = 0.0;
#pragma unroll 4
    for (int k = 4 * ((int)threadIdx.x & 31); k < K; k += 128) {
        const float4 a = row_piece(x, k, K, true), b = row_piece(w, k, K, true);
        s += ((double)a.x * b.x + (double)a.y * b.y) + ((double)a.z * b.z + (double)a.w * b.w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return (float)s;
}

template <bool SMALL>
__global__ void __launch_bounds__(Shape<SMALL>::THREADS, 1)
gemm_nt_f32_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, Args g) {
    using Sh = Shape<SMALL>;
    constexpr int THREADS = Sh::THREADS, COLS = Sh::COLS, X_PIECES = Sh::X_PIECES, X_ROWS = Sh::X_ROWS, STAGES = Sh::STAGES;
    constexpr unsigned TMEM = 512;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int nt = g.nt, plane_bytes = nt * CHUNK * 2;
    unsigned char* w_raw = smem;                                   // STAGES x [two halves][128 rows][32 values]; the sums at the end
    unsigned char* planes = w_raw + STAGES * W_CHUNK;              // STAGES x [three pieces][nt rows][128 bytes]
    Barriers* bar = reinterpret_cast<Barriers*>(planes + STAGES * PIECES * plane_bytes);
    volatile int* abort_flag = &bar->abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3;
    const int rank = (int)blockIdx.z;                              // segment
    // (the tiles of the same weight rows follow one another)
    const int m_tiles = (g.M + nt - 1) / nt, m0 = (int)(blockIdx.x % (unsigned)m_tiles) * nt, n0 = (int)(blockIdx.x / (unsigned)m_tiles) * BM;
    const int chunk0 = rank * g.segment_chunks, chunks = min(g.segment_chunks, (g.K + CHUNK - 1) / CHUNK - chunk0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&bar->w_full[s], 1);
            mbar_init(&bar->ready[s], Sh::W_WARPS + Sh::X_EACH + Sh::SUM_WARPS);
            mbar_init(&bar->done[s], 1);
        }
        bar->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == Sh::ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bar->tmem_base)), "r"(TMEM));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = bar->tmem_base, tmem_acc = tmem + STAGES * A_COLS;

    if (warp < Sh::W_WARPS) {
        // ------------------------------------------------------------------ the weights' pieces: half a chunk a warp
        const int half = warp >> 2, row = quarter * 32 + lane;
        const unsigned mine = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(half * 16);
        for (int c = 0; c < chunks; ++c) {
            const int b = c % STAGES;
            if (!mbar_wait(&bar->w_full[b], (unsigned)(c / STAGES) & 1, abort_flag, 1)) break;
            const unsigned char* src = w_raw + b * W_CHUNK + half * W_HALF + row * 128;
            float4 f[2][4];
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) f[q][i] = *reinterpret_cast<const float4*>(src + (((q * 4 + i) ^ (row & 7)) << 4));
            // (the instructions that read these columns are through: the copy waited for them)
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int q = 0; q < 2; ++q) split16_to_tmem<true>(f[q], mine + (unsigned)(b * A_COLS + q * 8), CHUNK / 2);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->ready[b]);
        }
    } else if (warp < Sh::FIRST_SUM) {
        // ------------------------------------------------------------------ the pieces of A's rows: eight lanes a row, the next chunk's values on their way
        pdl_wait();
        const int set = (warp - Sh::W_WARPS) / Sh::X_EACH, t = ((int)threadIdx.x - Sh::W_WARPS * 32) % (Sh::X_EACH * 32), row0 = t >> 3, q = t & 7;      // rows row0 + X_ROWS j
        const float* src = g.A + (size_t)(m0 + row0) * g.lda + (size_t)chunk0 * CHUNK + 8 * q;
        float4 f[X_PIECES][2];
        auto fetch = [&](int c) {
            const int left = c < chunks ? g.K - (chunk0 + c) * CHUNK - 8 * q : 0;      // values of the row from here on
#pragma unroll
            for (int j = 0; j < X_PIECES; ++j) {
                f[j][0] = f[j][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (X_ROWS * j + row0 >= nt || m0 + row0 + X_ROWS * j >= g.M) continue;
                const float* p = src + (size_t)(X_ROWS * j) * g.lda + c * CHUNK;
                if (left >= 8) {
                    f[j][0] = reinterpret_cast<const float4*>(p)[0];
                    f[j][1] = reinterpret_cast<const float4*>(p)[1];
                } else if (left > 0) {
                    f[j][0] = row_piece(p, 0, left, true);
                    f[j][1] = row_piece(p, 4, left, true);
                }
            }
        };
        fetch(set);
        for (int c = set; c < chunks; c += Sh::X_SETS) {
            const int b = c % STAGES;
            if (!mbar_wait(&bar->done[b], ((unsigned)(c / STAGES) & 1) ^ 1, abort_flag, 3)) break;
#pragma unroll
            for (int j = 0; j < X_PIECES; ++j) {
                const int row = row0 + X_ROWS * j;
                if (row < nt) split8_to_smem<true>(f[j][0], f[j][1], planes + b * PIECES * plane_bytes + row * 128 + ((q ^ (row & 7)) << 4), plane_bytes);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");           // the instructions read through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->ready[b]);
            fetch(c + Sh::X_SETS);                                       // (behind the fence, which would wait for it: 290 cycles against 46)
        }
    } else if (warp < Sh::ISSUER) {
        // ------------------------------------------------------------------ sums of a chunk into registers
        const int col0 = ((warp - Sh::FIRST_SUM) >> 2) * COLS, cols = min(COLS, nt - col0);
        const unsigned mine = tmem_acc + ((unsigned)(quarter * 32) << 16) + (unsigned)col0;
        float acc[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
        if (lane == 0) {                                           // both accumulators are free
            mbar_arrive(&bar->ready[0]);
            mbar_arrive(&bar->ready[1]);
        }
        for (int c = 0; c < chunks; ++c) {
            const int b = c & 1;
            if (!mbar_wait(&bar->done[c % STAGES], (unsigned)(c / STAGES) & 1, abort_flag, 4)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int j = 0; j < COLS; j += 16) {
                if (j >= cols) break;
                unsigned v[2][8];
                tmem_load8(mine + (unsigned)(b * nt + j), v[0]);
                if (j + 8 < COLS) tmem_load8(mine + (unsigned)(b * nt + j + 8), v[1]);     // (at most eight columns of the next tile of sums, not used)
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (j + e < COLS) acc[j + e] += __uint_as_float(v[e >> 3][e & 7]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->ready[(c + 2) % STAGES]);
        }
        // (all raw weights have been split when the last chunk's instructions are done: the sums may lie over them)
        float* part = reinterpret_cast<float*>(smem) + quarter * 32 + lane;        // [row of A][128 weight rows]
#pragma unroll
        for (int j = 0; j < COLS; ++j)
            if (j < cols) part[(col0 + j) * BM] = acc[j];
    } else if (warp == Sh::ISSUER) {
        // ------------------------------------------------------------------ the instructions
        const unsigned id = umma_idesc(BM, nt);
        for (int c = 0; c < chunks; ++c) {
            const int b = c % STAGES;
            const unsigned a = tmem + (unsigned)(b * A_COLS), d = tmem_acc + (unsigned)((c & 1) * nt);
            const unsigned long long x = umma_desc(planes + b * PIECES * plane_bytes), plane = (unsigned long long)(plane_bytes >> 4);
            if (!mbar_wait(&bar->ready[b], (unsigned)(c / STAGES) & 1, abort_flag, 5)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
#pragma unroll
                for (int i = 0; i < PAIRS; ++i)
#pragma unroll
                    for (int k = 0; k < CHUNK / UMMA_K; ++k)
                        umma_from_tmem(d, a + (unsigned)(BothUp::a(i) * (CHUNK / 2) + k * 8), x + BothUp::b(i) * plane + 2 * k, id, i > 0 || k > 0, k == 0 && BothUp::steps_down(i));
                umma_commit(&bar->done[b]);
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ raw weights.  The whole warp waits and an elected lane asks: in one lane's
        // branch a round of this took 1,350 cycles, and bounded everything.
        // (The kernel before may write what is taken for weights here: ahead of it goes only a request to have the first ones in L2.)
        if (elect_one())
            for (int c = 0; c < min(STAGES, chunks); ++c) {
                tma_prefetch_2d(&map_w, (chunk0 + c) * CHUNK, n0);
                tma_prefetch_2d(&map_w, (chunk0 + c) * CHUNK + 32, n0);
            }
        __syncwarp();
        pdl_wait();
        int c = 0;
        for (; c < chunks; ++c) {
            const int b = c % STAGES;
            if (!mbar_wait(&bar->done[b], ((unsigned)(c / STAGES) & 1) ^ 1, abort_flag, 2) || *abort_flag) break;
            if (elect_one()) {
                mbar_expect_tx(&bar->w_full[b], W_CHUNK);
                tma_load_2d(w_raw + b * W_CHUNK, &map_w, (chunk0 + c) * CHUNK, n0, &bar->w_full[b]);
                tma_load_2d(w_raw + b * W_CHUNK + W_HALF, &map_w, (chunk0 + c) * CHUNK + 32, n0, &bar->w_full[b]);
            }
            __syncwarp();
        }
        if (c < chunks)                                            // gave up: the copies that may still be in flight land first
            for (int j = max(0, c - STAGES); j < c; ++j)
                for (unsigned n = 0; n < WAIT_LIMIT && !mbar_try_wait(&bar->w_full[j % STAGES], (unsigned)(j / STAGES) & 1); ++n) {}
    }
    __syncwarp();
    pdl_launch_dependents();                                       // the next kernel may be scheduled while the sums are put together
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == Sh::ISSUER) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM));
    }
    if (g.segments > 1) cluster_sync();
    pdl_wait();
    // a share of the outputs over all segments in their order
    const unsigned part = smem_u32(smem);
    for (int e = rank * THREADS + (int)threadIdx.x; e < nt * (BM / 4); e += g.segments * THREADS) {
        const int m = m0 + e / (BM / 4), n = n0 + (e % (BM / 4)) * 4;      // (a warp has one row)
        if (m >= g.M) continue;
        float v[4];
        for (int from = 0; from < g.segments; ++from) {
            float4 f;
            const unsigned from_at = g.segments > 1 ? map_to_cta(part + 16u * (unsigned)e, (unsigned)from) : part + 16u * (unsigned)e;
            if (g.segments > 1)
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "r"(from_at) : "memory");
            else
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "r"(from_at) : "memory");
            if (from == 0) { v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; }
            else { v[0] += f.x; v[1] += f.y; v[2] += f.z; v[3] += f.w; }
        }
        bool off = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) off |= n + i < g.N && !isfinite(v[i]);
        if (__any_sync(0xffffffffu, off)) {
            const float* x = g.A + (size_t)m * g.lda;
            const bool nan = row_has_nan(x, g.K);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool again = n + i < g.N && !isfinite(v[i]);
                if (nan) { if (again) v[i] = __int_as_float(0x7fffffff); continue; }
                for (unsigned left = __ballot_sync(0xffffffffu, again); left; left &= left - 1) {
                    const int who = __ffs(left) - 1;
                    const float d = plain_dot(x, g.W + (size_t)(__shfl_sync(0xffffffffu, n, who) + i) * g.ldw, g.K);
                    if (lane == who) v[i] = d;
                }
            }
        }
        if (n >= g.N) continue;
        float* row = g.C + (size_t)m * g.ldc;
        if (g.vec_c && n + 4 <= g.N) *reinterpret_cast<float4*>(row + n) = make_float4(v[0], v[1], v[2], v[3]);
        else
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n + i < g.N) row[n + i] = v[i];
    }
    __syncwarp();
    if (g.segments > 1) cluster_sync();                            // nobody leaves while its sums are read
}

template <bool SMALL>
int launch(Args g, cudaStream_t stream) {
    CUtensorMap mw;
    if (int rc = make_map(&mw, g.W, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, g.N, g.K, g.ldw, BM, 32)) return rc;
    using Sh = Shape<SMALL>;
    auto bytes = [](int nt) { return 1024 + Sh::STAGES * (W_CHUNK + PIECES * (size_t)nt * CHUNK * 2) + sizeof(Barriers); };
    static_assert(1024 + Sh::STAGES * (W_CHUNK + PIECES * (size_t)Sh::MAXN * CHUNK * 2) + sizeof(Barriers) <= 232448 && Sh::MAXN * BM * 4 <= Sh::STAGES * W_CHUNK, "shared memory");
    const size_t most = bytes(Sh::MAXN), smem = bytes(g.nt);
    auto kernel = gemm_nt_f32_tcgen05_kernel<SMALL>;
    static LlmeGrants grants;
    if (cudaError_t e = llme_grant_smem(grants, kernel, most)) LLME_REFUSE("gemm_f32: cannot reserve %zu bytes of shared memory: %s", most, cudaGetErrorString(e));
    const long long blocks = (long long)((g.M + g.nt - 1) / g.nt) * ((g.N + BM - 1) / BM);
    if (blocks > 2147483647LL) LLME_REFUSE("gemm_f32: %d x %d outputs are too many for one launch", g.M, g.N);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks, 1, g.segments);
    cfg.blockDim = dim3(Shape<SMALL>::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = llme_pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = (unsigned)g.segments;
    cfg.attrs = attr;
    cfg.numAttrs = g.segments > 1 ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, mw, g);
    LLME_LAUNCH_STATUS();
}

// Which sizes: by K, N and the rows' alignment alone, never by M, so that a row's bits do not depend on the other rows.
bool takes(int N, int K, const void* A, const void* W, long long lda, long long ldw) {
    return K >= MIN_K && N >= MIN_N && ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && (lda | ldw) % 4 == 0;
}

// Segments: by K and N alone, 512 values and more each, at most five (larger clusters leave SMs unused), and as many as let few rows' blocks be on
// the GPU at once: one an SM.
// Rows of A a tile takes: few rows whole; else the tile with the least number of rounds times a block's time, in cycles: an instruction takes
// nt / 2, a chunk no less than its operands' splitting, and starting and the sums about 6,000.
int product(Args g, cudaStream_t stream) {
    const int all = (g.K + CHUNK - 1) / CHUNK, w_tiles = (g.N + BM - 1) / BM;
    int most = 148 / w_tiles;                                      // (of any device: the bits are not to depend on it)
    if (most > 5) most = 5;
    if (most > g.K / 512) most = g.K / 512;
    if (most < 1) most = 1;
    g.segment_chunks = (all + most - 1) / most;
    g.segments = (all + g.segment_chunks - 1) / g.segment_chunks;
    if (g.M <= 32) {
        g.nt = g.M <= 16 ? 16 : 32;
        return launch<true>(g, stream);
    }
    const long long others = (long long)w_tiles * g.segments;
    const int least = (g.M + Shape<false>::MAXN - 1) / Shape<false>::MAXN;
    double best = -1.0;
    for (int tiles = least; tiles <= least + 3; ++tiles) {
        const int nt = ((g.M + tiles - 1) / tiles + 15) / 16 * 16, blocks = (g.M + nt - 1) / nt;
        const double rounds = (double)((others * blocks + sm_count() - 1) / sm_count());
        const double cost = rounds * (g.segment_chunks * (12.0 * nt > 900.0 ? 12.0 * nt : 900.0) + 6000.0);
        if (best < 0.0 || cost < best) { best = cost; g.nt = nt; }
    }
    return launch<false>(g, stream);
}

}  // namespace split
