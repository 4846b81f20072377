// The grouped product of a mixture of experts on the tensor cores (bfloat16 operands, 32-bit sums): one product per
// expert over the (token, choice) pairs that were routed to it, rows gathered by token on the way in and scattered by
// pair on the way out where asked, silu(gate) * up (or max(., 0)^2 of a product without a gate) in the epilogue.
//
// A block owns a tile of BM pairs of ONE expert x BN output columns and walks K in steps of 32 through a cp.async
// pipeline of two or three stages; its four warps share the tile by columns (mma.sync m16n8k16, fragments by ldmatrix).
// Its shape is 64 x 64 (tiles of 128 rows on eight warps were no faster, 406 against
// 372 us for 2,048 tokens on 4 of 32 experts of 1,024: an expert's last tile is the emptier the larger the tiles are).
//
// Where experts get a few rows (decode steps) the weights are streamed instead (grouped_skinny_kernel): a block owns 16 weight rows
// of an expert (8 gate rows and the 8 up rows of the same outputs) as the M side of the instructions and up to 8 or 16 pairs as their
// N side; its eight warps take 64 values of k in turn, every operand goes from memory straight into the registers that the
// instruction reads (the order in which the products of a sum are added is free: four lanes take 8 consecutive values each), and
// four chunks a warp are on their way at a time.  Tiles of 16 x 128 through shared memory, three steps of 32 values of k in flight a block,
// took a mixture of 4 of 32 experts of 2,048 x 2,048 107 / 191 / 204 us at 2 / 8 / 24 tokens (the whole layer), this takes 54 / 110 / 164.
//
// The row tiles of all experts
// are numbered one after the other and a block finds its expert from the offsets; a launch has as many row tiles as
// any routing can need, and blocks beyond the step's own count leave at once.  A row's sums never depend on which
// other rows share its tile.
#include "common.cuh"
#include "kernel_args.h"

LLME_API const char* llme_last_error() { return llme_error_buffer(); }

namespace {

typedef __nv_bfloat16 bf16;
constexpr int BK = 32, LDS = BK + 8;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = valid ? 16 : 0;                     // 0: the 16 bytes are zero-filled and nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldmatrix_x4(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, const void* smem) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(a));
}
__device__ __forceinline__ void mma_bf16(float* d, const unsigned* a, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Row tile `tile` of all experts' tiles of BM rows, looked for by a whole warp (32 experts at a time: one after the other their
// offsets would be as many round trips to memory).
__device__ __forceinline__ bool find_tile(const int* __restrict__ offsets, int E, int BM, int tile, int lane, int* expert, int* first, int* rows) {
    int seen = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
        const int e = e0 + lane, lo = offsets[e < E ? e : E], n = offsets[e < E ? e + 1 : E] - lo, tiles = (n + BM - 1) / BM;
        int upto = tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const int at = tile - (seen + upto - tiles);
        const unsigned hit = __ballot_sync(0xffffffffu, at >= 0 && at < tiles);
        if (hit) {
            const int src = __ffs(hit) - 1, row = __shfl_sync(0xffffffffu, at, src) * BM, left = __shfl_sync(0xffffffffu, n, src) - row;
            *expert = e0 + src;
            *first = __shfl_sync(0xffffffffu, lo, src) + row;
            *rows = left < BM ? left : BM;
            return true;
        }
        seen += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

template <typename O> __device__ __forceinline__ void store2(O* p, float a, float b, bool two);
template <> __device__ __forceinline__ void store2<float>(float* p, float a, float b, bool two) {
    p[0] = a;
    if (two) p[1] = b;
}
template <> __device__ __forceinline__ void store2<bf16>(bf16* p, float a, float b, bool two) {
    p[0] = __float2bfloat16_rn(a);
    if (two) p[1] = __float2bfloat16_rn(b);
}

// BM x BN tile on WM x WNW warps, STAGES stages; ACT 1: the weight rows of a column are its gate row and, n_out further on, its up row;
// ACT 2: max(product, 0)^2 in the epilogue; ACT 3: gelu in its erf form.
template <int BM, int BN, int WM, int WNW, int STAGES, int ACT, typename O>
__global__ void __launch_bounds__(32 * WM * WNW) grouped_tc_kernel(LlmeGroupedArgs a) {
    constexpr int THREADS = 32 * WM * WNW, MT = BM / WM / 16, WN = BN / WNW, NT = WN / 8, HALVES = ACT == 1 ? 2 : 1;
    constexpr int A_STAGE = BM * LDS, B_STAGE = HALVES * BN * LDS;
    static_assert(MT >= 1 && NT >= 2 && NT % 2 == 0, "warp tiles are whole 16 x 16 pieces");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* As = reinterpret_cast<bf16*>(smem_raw);                      // [STAGES][BM][LDS]
    bf16* Bs = As + STAGES * A_STAGE;                                  // [STAGES][HALVES][BN][LDS]
    __shared__ int s_tile[3];
    __shared__ int s_src[BM], s_dst[BM];
    pdl_launch_dependents();
    pdl_wait();                                           // the offsets and the order come from the kernel before
    if (threadIdx.x < 32) {
        int e = -1, first = 0, rows = 0;
        if (!find_tile(a.offsets, a.num_experts, BM, blockIdx.y, threadIdx.x, &e, &first, &rows)) e = -1;
        if (threadIdx.x == 0) { s_tile[0] = e; s_tile[1] = first; s_tile[2] = rows; }
    }
    __syncthreads();
    const int e = s_tile[0], first = s_tile[1], rows = s_tile[2];
    if (e < 0) return;
    for (int r = threadIdx.x; r < BM; r += THREADS) {
        const int pair = r < rows ? a.order[first + r] : -1;
        s_src[r] = r < rows ? (a.gather ? pair / a.top_k : first + r) : -1;
        s_dst[r] = r < rows ? (a.scatter ? pair : first + r) : -1;
    }
    __syncthreads();
    const int n_out = ACT == 1 ? a.n / 2 : a.n;
    const int col0 = blockIdx.x * BN;
    const bf16* x = (const bf16*)a.x;
    const bf16* w = (const bf16*)a.w + (size_t)e * a.w_expert;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp / WNW, wn = warp % WNW;
    const int steps = (a.k + BK - 1) / BK;

    auto load_stage = [&](int stage, int step) {
        if (step < steps) {
            const int k0 = step * BK;
            for (int i = threadIdx.x; i < BM * (BK / 8); i += THREADS) {
                const int r = i / (BK / 8), c = (i % (BK / 8)) * 8;
                const int src = s_src[r];
                const bool ok = src >= 0 && k0 + c < a.k;
                cp_async16(As + stage * A_STAGE + r * LDS + c, ok ? x + (size_t)src * a.ldx + k0 + c : x, ok);
            }
            for (int i = threadIdx.x; i < HALVES * BN * (BK / 8); i += THREADS) {
                const int half = i / (BN * (BK / 8)), r = (i / (BK / 8)) % BN, c = (i % (BK / 8)) * 8;
                const bool ok = col0 + r < n_out && k0 + c < a.k;
                cp_async16(Bs + stage * B_STAGE + (half * BN + r) * LDS + c, ok ? w + (size_t)(half * n_out + col0 + r) * a.ldw + k0 + c : w, ok);
            }
        }
        cp_async_commit();                                // one group a step, also an empty one: the count below relies on it
    };

    float acc[HALVES][MT][NT][4];
#pragma unroll
    for (int h = 0; h < HALVES; ++h)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[h][m][n][i] = 0.0f;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) load_stage(s, s);
    for (int s = 0; s < steps; ++s) {
        cp_async_wait<STAGES - 2>();                      // the loads of step s have landed
        __syncthreads();                                  // ... for every thread, and step s - 1 has been read by all
        load_stage((s + STAGES - 1) % STAGES, s + STAGES - 1);
        const bf16* At = As + (s % STAGES) * A_STAGE + wm * (BM / WM) * LDS;
        const bf16* Bt = Bs + (s % STAGES) * B_STAGE;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 16) {
            unsigned af[MT][4];
#pragma unroll
            for (int m = 0; m < MT; ++m)
                ldmatrix_x4(af[m][0], af[m][1], af[m][2], af[m][3], At + (m * 16 + (lane & 15)) * LDS + kk + (lane >> 4) * 8);
#pragma unroll
            for (int h = 0; h < HALVES; ++h)
#pragma unroll
                for (int n = 0; n < NT; n += 2) {
                    unsigned b0, b1, b2, b3;              // (n-tile n: k 0-7, k 8-15), (n-tile n + 1: k 0-7, k 8-15)
                    ldmatrix_x4(b0, b1, b2, b3, Bt + (h * BN + wn * WN + n * 8 + (lane & 7) + (lane >> 4) * 8) * LDS + kk + ((lane >> 3) & 1) * 8);
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        mma_bf16(acc[h][m][n], af[m], b0, b1);
                        mma_bf16(acc[h][m][n + 1], af[m], b2, b3);
                    }
                }
        }
    }

    O* out = (O*)a.out;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int half_rows = 0; half_rows < 2; ++half_rows) {
            const int r = wm * (BM / WM) + m * 16 + (lane >> 2) + half_rows * 8;
            const int dst = s_dst[r];
            if (dst < 0) continue;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int col = col0 + wn * WN + n * 8 + (lane & 3) * 2;
                if (col >= n_out) continue;
                float v0 = acc[0][m][n][half_rows * 2], v1 = acc[0][m][n][half_rows * 2 + 1];
                if (ACT == 2) {
                    v0 = relu2(v0);
                    v1 = relu2(v1);
                }
                if (ACT == 3) {
                    v0 = gelu_erf(v0);
                    v1 = gelu_erf(v1);
                }
                if (ACT == 1) {
                    // gate and up pass through bfloat16 first, as they do when the activation is a kernel of its own
                    const float g0 = __bfloat162float(__float2bfloat16_rn(v0)), g1 = __bfloat162float(__float2bfloat16_rn(v1));
                    const float u0 = __bfloat162float(__float2bfloat16_rn(acc[HALVES - 1][m][n][half_rows * 2]));
                    const float u1 = __bfloat162float(__float2bfloat16_rn(acc[HALVES - 1][m][n][half_rows * 2 + 1]));
                    v0 = silu_mul_bf16(g0, u0);
                    v1 = silu_mul_bf16(g1, u1);
                }
                store2<O>(out + (size_t)dst * a.ldo + col, v0, v1, col + 1 < n_out);
            }
        }
}

// Few rows an expert.  MT: 8-pair tiles (a tile of 8 MT pairs of one expert).
constexpr int KC = 64, SKINNY_WARPS = 8, UNROLL = 4;

// weights are read by few blocks: do not keep them in L1
__device__ __forceinline__ uint4 load_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

template <int MT, int ACT, typename O>
__global__ void __launch_bounds__(32 * SKINNY_WARPS, 2) grouped_skinny_kernel(LlmeGroupedArgs a) {
    constexpr int BM = 8 * MT;
    __shared__ float red[SKINNY_WARPS][BM][16];
    __shared__ int s_tile[3], s_dst[BM];
    pdl_launch_dependents();
    pdl_wait();                                           // the offsets and the order come from the kernel before
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3, r = lane >> 2;
    if (warp == 0) {
        int e = -1, first = 0, rows = 0;
        if (!find_tile(a.offsets, a.num_experts, BM, blockIdx.y, lane, &e, &first, &rows)) e = -1;
        if (lane == 0) { s_tile[0] = e; s_tile[1] = first; s_tile[2] = rows; }
    }
    __syncthreads();
    const int e = s_tile[0], first = s_tile[1], rows = s_tile[2];
    if (e < 0) return;
    const int n_out = ACT == 1 ? a.n / 2 : a.n, rg = blockIdx.x;
    // the pairs of this lane (pair lane / 4 of every tile of eight) and the weight rows (clamped: a row past the end is read, not stored)
    const bf16* xr[MT];
    bool xok[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        xok[m] = m * 8 + r < rows;
        const int at = first + (xok[m] ? m * 8 + r : 0), pair = a.order[at];
        xr[m] = (const bf16*)a.x + (size_t)(a.gather ? pair / a.top_k : at) * a.ldx + quad * 8;
        if (warp == 0 && quad == 0) s_dst[m * 8 + r] = a.scatter ? pair : at;
    }
    const int row0 = ACT == 1 ? min(rg * 8 + r, n_out - 1) : min(rg * 16 + r, n_out - 1);
    const int row1 = ACT == 1 ? n_out + row0 : min(rg * 16 + r + 8, n_out - 1);
    const bf16* w = (const bf16*)a.w + (size_t)e * a.w_expert;
    const bf16* w0 = w + (size_t)row0 * a.ldw + quad * 8;
    const bf16* w1 = w + (size_t)row1 * a.ldw + quad * 8;
    float acc[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.0f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const int chunks = (a.k + KC - 1) / KC;
    for (int c = warp; c < chunks; c += UNROLL * SKINNY_WARPS) {
        uint4 wa[UNROLL][2], wb[UNROLL][2], xv[UNROLL][MT][2];
#pragma unroll
        for (int q = 0; q < UNROLL; ++q)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int k = (c + q * SKINNY_WARPS) * KC + b * 32;
                const bool ok = k + quad * 8 < a.k;       // k is a multiple of 8: a piece is inside or outside
                wa[q][b] = ok ? load_stream(w0 + k) : zero;
                wb[q][b] = ok ? load_stream(w1 + k) : zero;
#pragma unroll
                for (int m = 0; m < MT; ++m) xv[q][m][b] = ok && xok[m] ? *reinterpret_cast<const uint4*>(xr[m] + k) : zero;
            }
#pragma unroll
        for (int q = 0; q < UNROLL; ++q)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const unsigned lo[4] = {wa[q][b].x, wb[q][b].x, wa[q][b].y, wb[q][b].y}, hi[4] = {wa[q][b].z, wb[q][b].z, wa[q][b].w, wb[q][b].w};
                    mma_bf16(acc[m], lo, xv[q][m][b].x, xv[q][m][b].y);
                    mma_bf16(acc[m], hi, xv[q][m][b].z, xv[q][m][b].w);
                }
    }
    // the warps' partial sums, added in a fixed order
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) red[warp][m * 8 + quad * 2 + (i & 1)][r + (i >> 1) * 8] = acc[m][i];
    __syncthreads();
    auto total = [&](int tok, int row) {
        float v = red[0][tok][row];
#pragma unroll
        for (int wp = 1; wp < SKINNY_WARPS; ++wp) v += red[wp][tok][row];
        return v;
    };
    constexpr int COLS = ACT == 1 ? 8 : 16;
    for (int i = threadIdx.x; i < BM * COLS; i += 32 * SKINNY_WARPS) {
        const int tok = i / COLS, j = i % COLS, col = rg * COLS + j;
        if (tok >= rows || col >= n_out) continue;
        float v = total(tok, j);
        if (ACT == 1)                                     // gate and up pass through bfloat16 first, as they do when the activation is a kernel of its own
            v = silu_mul_bf16(__bfloat162float(__float2bfloat16_rn(v)), __bfloat162float(__float2bfloat16_rn(total(tok, j + 8))));
        if (ACT == 2) v = relu2(v);
        if (ACT == 3) v = gelu_erf(v);
        reinterpret_cast<O*>(a.out)[(size_t)s_dst[tok] * a.ldo + col] = from_f32<O>(v);
    }
}

// Row tiles of BM pairs that any routing can need: every expert may add one that is not full.
int most_tiles(const LlmeGroupedArgs& a, int BM) {
    const int most = a.num_experts < a.pairs ? a.num_experts : a.pairs, tiles = (a.pairs + BM - 1) / BM + most;
    return tiles < a.pairs ? tiles : a.pairs;
}

template <int MT, int ACT, typename O>
int launch_skinny(const LlmeGroupedArgs& a, cudaStream_t s) {
    const int tiles = most_tiles(a, 8 * MT), cols = ACT == 1 ? 8 : 16, n_out = ACT == 1 ? a.n / 2 : a.n;
    if (tiles > 65535) LLME_REFUSE("grouped_linear_tc: %d row tiles exceed a launch", tiles);
    llme_launch(grouped_skinny_kernel<MT, ACT, O>, dim3((n_out + cols - 1) / cols, tiles), dim3(32 * SKINNY_WARPS), 0, s, a);
    LLME_LAUNCH_STATUS();
}

template <int BM, int BN, int WM, int WNW, int STAGES, int ACT, typename O>
int launch(const LlmeGroupedArgs& a, cudaStream_t s) {
    constexpr int SMEM = STAGES * (BM + (ACT == 1 ? 2 : 1) * BN) * LDS * (int)sizeof(bf16);
    const int n_out = ACT == 1 ? a.n / 2 : a.n;
    const int tiles = most_tiles(a, BM);
    if (tiles > 65535) {
        snprintf(llme_error_buffer(), 512, "grouped_linear_tc: %d row tiles exceed a launch", tiles);
        return -1;
    }
    auto kernel = grouped_tc_kernel<BM, BN, WM, WNW, STAGES, ACT, O>;
    static LlmeGrants grants;
    if (SMEM > 48 * 1024 && llme_grant_smem(grants, kernel, SMEM) != cudaSuccess) LLME_REFUSE("grouped_linear_tc: %d bytes of shared memory are not available", SMEM);
    llme_launch(kernel, dim3((n_out + BN - 1) / BN, tiles), dim3(32 * WM * WNW), (size_t)SMEM, s, a);
    LLME_LAUNCH_STATUS();
}

// Rows an expert in the mean (the routing itself is on the device): tiles of 8 pairs, of 16, or of 64 through shared memory.  (From 4 rows on,
// and below where that is estimated to be faster, the tcgen05 kernel serves what it can; without it 16-pair tiles take that mixture 266 us at 124 tokens and 327 us at 160, 64-pair
// tiles 279 us at 400.)
constexpr long long SKINNY_8 = 4, SKINNY_16 = 16;

template <int ACT, typename O>
int dispatch(const LlmeGroupedArgs& a, cudaStream_t s) {
    if ((long long)a.pairs <= SKINNY_8 * a.num_experts) return launch_skinny<1, ACT, O>(a, s);
    if ((long long)a.pairs < SKINNY_16 * a.num_experts) return launch_skinny<2, ACT, O>(a, s);
    return launch<64, 64, 1, 4, 3, ACT, O>(a, s);
}

}  // namespace

LLME_API int llme_grouped_linear_tc(const LlmeGroupedArgs* args, int x_dtype, int w_dtype, int out_dtype, cudaStream_t stream) {
    const LlmeGroupedArgs& a = *args;
    if (a.pairs <= 0 || a.n <= 0) return 0;
    if (!a.x || !a.w || !a.out || !a.offsets || !a.order) LLME_REFUSE("grouped_linear_tc: null pointer");
    if (x_dtype != LLME_BF16 || w_dtype != LLME_BF16) LLME_REFUSE("grouped_linear_tc: bfloat16 operands only");
    if (a.num_experts <= 0 || a.top_k <= 0 || a.k <= 0 || a.act < 0 || a.act > 3 || (a.act == 1 && a.n % 2)) LLME_REFUSE("grouped_linear_tc: bad size");
    if (a.k % 8 || a.ldx % 8 || a.ldw % 8 || a.w_expert % 8 || (((uintptr_t)a.x | (uintptr_t)a.w) & 15))
        LLME_REFUSE("grouped_linear_tc: rows must be whole 16-byte pieces");
    if (out_dtype == LLME_BF16) return a.act == 1 ? dispatch<1, bf16>(a, stream) : a.act == 2 ? dispatch<2, bf16>(a, stream) : a.act == 3 ? dispatch<3, bf16>(a, stream) : dispatch<0, bf16>(a, stream);
    if (out_dtype == LLME_F32) return a.act == 1 ? dispatch<1, float>(a, stream) : a.act == 2 ? dispatch<2, float>(a, stream) : a.act == 3 ? dispatch<3, float>(a, stream) : dispatch<0, float>(a, stream);
    LLME_REFUSE("grouped_linear_tc: unsupported output dtype %d", out_dtype);
}
