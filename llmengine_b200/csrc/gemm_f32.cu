// True 32-bit matrix product C[M,N] = A[M,K] * W[N,K]^T.  It is the matrix product of the whole 32-bit path and the plain twin that the
// tensor-core kernels are checked against.  Float weights whose rows begin on 16 bytes go to the tensor cores in pieces that keep all 24
// bits (gemm_f32_tcgen05.cuh); everything else (bfloat16 weights, batches of products, fewer than 512 values, odd row strides) is multiplied
// and added on the CUDA cores, in the forms below.
//
// K is cut into S segments of equal length, S = K / 1024 between 1 and 8; every output element adds the products of a
// segment in the order of k, and then the segments' sums in their order.  S depends on K alone, so a row's result does not
// depend on how many other rows are in the launch, whichever of the forms below serves it:
//
//   * a block walks all segments of its tile and adds each to C;
//   * a cluster of S blocks, one segment each: the blocks leave their sums in shared memory, and each adds a share of the tile
//     over the blocks in their order.  It fills the GPU where the tiles alone do not (300 x 2048 has 80 tiles of 64 x 128).
//
// 16 x 16 threads hold TM x TN outputs each, as packed pairs of neighbouring columns (fma.rn.f32x2: one instruction, each half
// rounds as fmaf does); operands lie in shared memory k by k, two stages, the next one on its way through registers.
// Bound by shared memory, whose path is 87 to 89 % busy while the multiply-adds fill 55 % of theirs.  All figures of this file are of float weights,
// taken when these forms served them too: 300 x 11008 x 2048 took 376 us and 300 x 2048 x 5504 206 us (36 and 33 TFLOP/s of 74; 2,048 rows: 50 and
// 44); one block per 64 x 64 tile with 4 x 4 outputs a thread, whatever the shape, took 675 and 617 us.
// Up to 32 rows a third form streams the weights (further down).
//
// Reference counterparts: sgemm_nt_kernel (src/runtime/kernels/cuda_kernels.cu:282-294,
// one thread per output, no tiling) and the cublasSgemm call of sgemm_nt_cublas (:892-908).
#include <cuda.h>

#include "common.cuh"

LLME_API const char* llme_last_error() { return llme_error_buffer(); }

namespace {

constexpr int BK = 16, THREADS = 256, MAX_SEGMENTS = 8;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
// values k .. k + 3 of a row, zeros from `end` on
template <typename T>
__device__ __forceinline__ float4 row_piece(const T* row, int k, int end, bool vec) {
    if (vec && k + 4 <= end) return load4(row + k);
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (k < end) v.x = to_f32(row[k]);
    if (k + 1 < end) v.y = to_f32(row[k + 1]);
    if (k + 2 < end) v.z = to_f32(row[k + 2]);
    if (k + 3 < end) v.w = to_f32(row[k + 3]);
    return v;
}

template <typename WT>
struct Problem {
    const float* A; const WT* W; float* C;
    int M, N, K, segment, segments, vec_a, vec_w, vec_c;
    long long lda, ldw, ldc, sa, sw, sc;
};

// The i-th of a thread's T rows (or columns) of a tile: four side by side, the next four 64 further on.
template <int T> __device__ __forceinline__ int place(int t, int i) { return T == 1 ? t : (i / 4) * 64 + t * 4 + (i & 3); }

template <int TM, int TN>
struct Tile {
    static constexpr int BM = 16 * TM, BN = 16 * TN;
    float a[2][BK][BM + 4], w[2][BK][BN + 4];
};

template <typename WT, int TM, int TN, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 2) gemm_nt_f32_kernel(Problem<WT> g) {
    constexpr int BM = 16 * TM, BN = 16 * TN, AL = (BM * BK / 4 + THREADS - 1) / THREADS, WL = BN * BK / 4 / THREADS;
    static_assert(WL >= 1 && TN % 4 == 0, "a tile has at least 64 columns");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Tile<TM, TN>& sm = *reinterpret_cast<Tile<TM, TN>*>(smem_raw);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int member = SPLIT ? (int)blockIdx.z / g.segments : (int)blockIdx.z, rank = SPLIT ? (int)blockIdx.z % g.segments : 0;
    const float* A = g.A + (size_t)member * g.sa;          // one member of a batch of products
    const WT* W = g.W + (size_t)member * g.sw;
    float* C = g.C + (size_t)member * g.sc;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const bool vec_a = g.vec_a, vec_w = g.vec_w;

    f32x2 acc[TM][TN / 2];
    for (int seg = SPLIT ? rank : 0; seg < (SPLIT ? rank + 1 : g.segments); ++seg) {
        const int k_begin = seg * g.segment, k_end = min(g.K, k_begin + g.segment);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
        float4 pa[AL], pw[WL];
        auto fetch = [&](int k0) {
#pragma unroll
            for (int i = 0; i < AL; ++i) {
                const int e = tid + i * THREADS, r = e >> 2, k = k0 + (e & 3) * 4;
                pa[i] = e < BM * BK / 4 && m0 + r < g.M ? row_piece(A + (size_t)(m0 + r) * g.lda, k, k_end, vec_a) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int i = 0; i < WL; ++i) {
                const int e = tid + i * THREADS, r = e >> 2, k = k0 + (e & 3) * 4;
                pw[i] = n0 + r < g.N ? row_piece(W + (size_t)(n0 + r) * g.ldw, k, k_end, vec_w) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        };
        auto put = [&](int s) {
#pragma unroll
            for (int i = 0; i < AL; ++i) {
                const int e = tid + i * THREADS, r = e >> 2, k = (e & 3) * 4;
                if (e < BM * BK / 4) {
                    sm.a[s][k][r] = pa[i].x; sm.a[s][k + 1][r] = pa[i].y; sm.a[s][k + 2][r] = pa[i].z; sm.a[s][k + 3][r] = pa[i].w;
                }
            }
#pragma unroll
            for (int i = 0; i < WL; ++i) {
                const int e = tid + i * THREADS, r = e >> 2, k = (e & 3) * 4;
                sm.w[s][k][r] = pw[i].x; sm.w[s][k + 1][r] = pw[i].y; sm.w[s][k + 2][r] = pw[i].z; sm.w[s][k + 3][r] = pw[i].w;
            }
        };
        fetch(k_begin);
        put(0);
        __syncthreads();
        int s = 0;
        for (int k0 = k_begin; k0 < k_end; k0 += BK, s ^= 1) {
            const bool more = k0 + BK < k_end;
            if (more) fetch(k0 + BK);
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a[TM];
                f32x2 w[TN / 2];
                if (TM == 1) a[0] = sm.a[s][kk][ty];
                else
#pragma unroll
                    for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(&a[i]) = *reinterpret_cast<const float4*>(&sm.a[s][kk][place<TM>(ty, i)]);
#pragma unroll
                for (int j = 0; j < TN; j += 4) {
                    const ulonglong2 two = *reinterpret_cast<const ulonglong2*>(&sm.w[s][kk][place<TN>(tx, j)]);
                    w[j / 2] = two.x;
                    w[j / 2 + 1] = two.y;
                }
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const f32x2 aa = pack2(a[i], a[i]);
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(aa, w[j], acc[i][j]);
                }
            }
            if (more) put(s ^ 1);
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < (SPLIT ? 0 : TM); ++i) {
            const int gm = m0 + place<TM>(ty, i);
            if (gm >= g.M) continue;
            float* row = C + (size_t)gm * g.ldc;
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
                const int gn = n0 + place<TN>(tx, j);
                float v[4];
                unpack2(acc[i][j / 2], v[0], v[1]);
                unpack2(acc[i][j / 2 + 1], v[2], v[3]);
                if (g.vec_c && gn + 4 <= g.N) {
                    float4 o = make_float4(v[0], v[1], v[2], v[3]);
                    if (seg > 0) {
                        const float4 c = *reinterpret_cast<const float4*>(row + gn);
                        o = make_float4(c.x + o.x, c.y + o.y, c.z + o.z, c.w + o.w);
                    }
                    *reinterpret_cast<float4*>(row + gn) = o;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (gn + e < g.N) row[gn + e] = seg > 0 ? row[gn + e] + v[e] : v[e];
                }
            }
        }
    }
    if (SPLIT) {
        // this block's sums into its shared memory, then a share of the tile's rows over all blocks in their order
        float* part = reinterpret_cast<float*>(smem_raw);  // [BM][BN] (the stages are done with)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
                float4 o;
                unpack2(acc[i][j / 2], o.x, o.y);
                unpack2(acc[i][j / 2 + 1], o.z, o.w);
                *reinterpret_cast<float4*>(part + place<TM>(ty, i) * BN + place<TN>(tx, j)) = o;
            }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const unsigned mine = (unsigned)__cvta_generic_to_shared(part);
        for (int e = rank * THREADS + tid; e < BM * BN / 4; e += g.segments * THREADS) {
            float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int from = 0; from < g.segments; ++from) {
                unsigned at;
                float4 v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine + 16u * (unsigned)e), "r"(from));
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
                sum = from == 0 ? v : make_float4(sum.x + v.x, sum.y + v.y, sum.z + v.z, sum.w + v.w);
            }
            const int gm = m0 + e / (BN / 4), gn = n0 + (e % (BN / 4)) * 4;
            if (gm >= g.M) continue;
            float* row = C + (size_t)gm * g.ldc;
            if (g.vec_c && gn + 4 <= g.N) *reinterpret_cast<float4*>(row + gn) = sum;
            else {
                if (gn < g.N) row[gn] = sum.x;
                if (gn + 1 < g.N) row[gn + 1] = sum.y;
                if (gn + 2 < g.N) row[gn + 2] = sum.z;
                if (gn + 3 < g.N) row[gn + 3] = sum.w;
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");     // nobody leaves while its sums are read
    }
}

template <typename WT, int TM, int TN, bool SPLIT>
int launch(const Problem<WT>& g, int batch, cudaStream_t stream) {
    constexpr int BM = 16 * TM, BN = 16 * TN;
    constexpr size_t stages = sizeof(Tile<TM, TN>), part = SPLIT ? (size_t)BM * BN * 4 : 0, smem = stages > part ? stages : part;
    auto kernel = gemm_nt_f32_kernel<WT, TM, TN, SPLIT>;
    static LlmeGrants grants;
    if (cudaError_t e = llme_grant_smem(grants, kernel, smem)) LLME_REFUSE("gemm_f32: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((g.N + BN - 1) / BN, (g.M + BM - 1) / BM, SPLIT ? batch * g.segments : batch);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)g.segments;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, g);
    LLME_LAUNCH_STATUS();
}

__device__ __forceinline__ float4 load4_shared(const unsigned char* p, float) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4_shared(const unsigned char* p, __nv_bfloat16) { return load4(reinterpret_cast<const __nv_bfloat16*>(p)); }
// `bytes` of SIZE from src, zeros behind them
template <int SIZE>
__device__ __forceinline__ void copy_async(unsigned char* dst, const void* src, int bytes) {
    const unsigned at = (unsigned)__cvta_generic_to_shared(dst);
    if (SIZE == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(src), "r"(bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(at), "l"(src), "r"(bytes) : "memory");
}

// A few rows: the weights are streamed.  A block serves 16 weight rows and MT rows of A; each of its warps walks one segment of K,
// 32 values at a time, through copies of its own (no barrier until the segments are added, in their order).  A lane has R weight
// rows and T rows of A, and each of its outputs is one chain of multiply-adds in the order of k, as in the tiles.
// One row is bound by the weights and the chains' latency, 16 rows by the warps' issue (16 weight rows a block is what gives 2,048
// outputs enough blocks).  Against the tiles, whose steps of 16 values each wait for a barrier (11008 x 2048 / 2048 x 5504, us):
// 1 row 21 / 19 and 117 / 66, 8 rows 31 / 25 and 117 / 66, 16 rows 45 / 35 and 118 / 67, 32 rows 73 / 50 and 119 / 74.
constexpr int FEW_N = 16, FEW_K = 32, FEW_ROWS = 32;
__host__ __device__ constexpr int few_stages(int mt) { return mt <= 4 ? 6 : mt <= 16 ? 5 : 4; }
template <typename WT, int MT>
__host__ __device__ constexpr int few_stage_bytes() { return FEW_N * FEW_K * (int)sizeof(WT) + MT * FEW_K * 4; }

template <typename WT, int MT>
__global__ void gemm_few_f32_kernel(Problem<WT> g) {
    constexpr int R = MT <= 4 ? 1 : MT <= 16 ? 2 : 4, RG = FEW_N / R, TG = 32 / RG, T = MT / TG;     // a lane's R x T outputs
    constexpr int STAGES = few_stages(MT), WB = FEW_N * FEW_K * (int)sizeof(WT), STAGE = few_stage_bytes<WT, MT>();
    constexpr int PIECE = 4 * (int)sizeof(WT);             // four weights
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rg = lane % RG, tg = lane / RG;
    const float* A = g.A + (size_t)blockIdx.z * g.sa;
    const WT* W = g.W + (size_t)blockIdx.z * g.sw;
    float* C = g.C + (size_t)blockIdx.z * g.sc;
    const int n0 = blockIdx.x * FEW_N, m0 = blockIdx.y * MT;
    const int k_begin = warp * g.segment, k_end = min(g.K, k_begin + g.segment), chunks = (k_end - k_begin + FEW_K - 1) / FEW_K;
    unsigned char* mine = smem_raw + (size_t)warp * STAGES * STAGE;
    // where a row's p-th four values lie: the lanes of one shared-memory pass (8 of 16 bytes, 16 of 8) meet every bank once
    auto place_w = [](int r, int p) { return (r * 8 + (p ^ ((sizeof(WT) == 4 ? r : r >> 1) & 7))) * PIECE; };
    auto place_a = [](int r, int p) { return (r * 8 + (p ^ (r & 7))) * 16; };
    auto request = [&](int c, int stage) {
        if (c < chunks) {
            unsigned char* at = mine + stage * STAGE;
            const int k0 = k_begin + c * FEW_K + (lane & 7) * 4, some = max(0, min(4, k_end - k0));
#pragma unroll
            for (int i = 0; i < FEW_N / 4; ++i) {
                const int r = i * 4 + (lane >> 3), n = n0 + r < g.N ? some : 0;
                copy_async<PIECE>(at + place_w(r, lane & 7), n ? W + (size_t)(n0 + r) * g.ldw + k0 : W, n * (int)sizeof(WT));
            }
#pragma unroll
            for (int i = 0; i < (MT + 3) / 4; ++i) {
                const int r = i * 4 + (lane >> 3), n = m0 + r < g.M ? some : 0;
                if (r < MT) copy_async<16>(at + WB + place_a(r, lane & 7), n ? A + (size_t)(m0 + r) * g.lda + k0 : A, n * 4);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[R][T];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int t = 0; t < T; ++t) acc[i][t] = 0.0f;
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) request(c, c);
    int stage = 0;
    for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncwarp();                                      // every lane's copies are there, and the stage before this one is read
        request(c + STAGES - 1, stage == 0 ? STAGES - 1 : stage - 1);
        const unsigned char* at = mine + stage * STAGE;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            float4 w[R];
#pragma unroll
            for (int i = 0; i < R; ++i) w[i] = load4_shared(at + place_w(rg + i * RG, p), WT());
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const float4 v = *reinterpret_cast<const float4*>(at + WB + place_a(tg + t * TG, p));
#pragma unroll
                for (int i = 0; i < R; ++i) acc[i][t] = fmaf(v.w, w[i].w, fmaf(v.z, w[i].z, fmaf(v.y, w[i].y, fmaf(v.x, w[i].x, acc[i][t]))));
            }
        }
        stage = stage == STAGES - 1 ? 0 : stage + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    float* part = reinterpret_cast<float*>(mine);          // [MT][16], this segment's sums
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int t = 0; t < T; ++t) part[(tg + t * TG) * FEW_N + rg + i * RG] = acc[i][t];
    __syncthreads();
    for (int e = threadIdx.x; e < MT * FEW_N; e += blockDim.x) {
        const int m = m0 + e / FEW_N, n = n0 + e % FEW_N;
        if (m >= g.M || n >= g.N) continue;
        float sum = 0.0f;
        for (int from = 0; from < g.segments; ++from) {
            const float v = reinterpret_cast<const float*>(smem_raw + (size_t)from * STAGES * STAGE)[e];
            sum = from == 0 ? v : sum + v;
        }
        C[(size_t)m * g.ldc + n] = sum;
    }
}

template <typename WT, int MT>
int launch_few(const Problem<WT>& g, int batch, cudaStream_t stream) {
    constexpr int one = few_stages(MT) * few_stage_bytes<WT, MT>();
    auto kernel = gemm_few_f32_kernel<WT, MT>;
    static LlmeGrants grants;
    if (cudaError_t e = llme_grant_smem(grants, kernel, MAX_SEGMENTS * one))
        LLME_REFUSE("gemm_f32: cannot reserve %d bytes of shared memory: %s", MAX_SEGMENTS * one, cudaGetErrorString(e));
    kernel<<<dim3((g.N + FEW_N - 1) / FEW_N, (g.M + MT - 1) / MT, batch), g.segments * 32, g.segments * one, stream>>>(g);
    LLME_LAUNCH_STATUS();
}

int sm_count() {
    static int n = [] {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) v = 148;
        return v;
    }();
    return n;
}

// Which tile, and whether a cluster shares its segments: the least number of rounds times a block's work.  A block's rate relative to
// that of 128 x 128 outputs (`rate`): what its operands cost beside the multiply-adds (two 16-byte loads from shared memory for 64 of
// them, one and a quarter for 8).  A round is a block an SM, although two find room there: two share its multiply-adds and its shared
// memory.  The 64 and 32 values of k stand for a cluster's and a further segment's sums.  All of it is an estimate: over 90 sizes (33 to
// 2,048 rows on 512 to 11,008 outputs of 600 to 5,504 values) its choice is within 5 % of the best of the eight forms in 82, and
// at worst 23 % behind (256 x 2048 x 5504: 251 us against 204); 300 x 11008 x 2048 takes 376 us so, 365 at best, 402 in tiles of 128.
template <typename WT>
int dispatch(const Problem<WT>& g, int batch, cudaStream_t stream) {
    const int bm[4] = {128, 64, 64, 16}, bn[4] = {128, 128, 64, 128};
    const double rate[4] = {1.0, 0.9, 0.75, 0.3};
    int best = -1;
    double best_cost = 0.0;
    for (int i = 0; i < 8; ++i) {
        const int c = i >> 1, split = i & 1;
        if (split && (g.segments == 1 || (long long)batch * g.segments > 65535)) continue;
        if ((g.M + bm[c] - 1) / bm[c] > 65535) continue;
        const long long tiles = (long long)((g.M + bm[c] - 1) / bm[c]) * ((g.N + bn[c] - 1) / bn[c]) * batch, blocks = split ? tiles * g.segments : tiles;
        const double rounds = (double)((blocks + sm_count() - 1) / sm_count());
        const double cost = rounds * bm[c] * bn[c] * (split ? g.segment + 64.0 : (double)g.K + 32.0 * g.segments) / rate[c];
        if (best < 0 || cost < best_cost) { best = i; best_cost = cost; }
    }
    switch (best) {
        case 0: return launch<WT, 8, 8, false>(g, batch, stream);
        case 1: return launch<WT, 8, 8, true>(g, batch, stream);
        case 2: return launch<WT, 4, 8, false>(g, batch, stream);
        case 3: return launch<WT, 4, 8, true>(g, batch, stream);
        case 4: return launch<WT, 4, 4, false>(g, batch, stream);
        case 5: return launch<WT, 4, 4, true>(g, batch, stream);
        case 6: return launch<WT, 1, 8, false>(g, batch, stream);
        case 7: return launch<WT, 1, 8, true>(g, batch, stream);
    }
    LLME_REFUSE("gemm_f32: M = %d needs more than 65535 grid rows", g.M);
}

#include "gemm_f32_tcgen05.cuh"

template <typename WT>
int product(const float* A, const WT* W, float* C, int M, int N, int K, long long lda, long long ldw, long long ldc, int batch, long long sa,
            long long sw, long long sc, cudaStream_t stream) {
    Problem<WT> g = {A, W, C, M, N, K, 0, 0, 0, 0, 0, lda, ldw, ldc, sa, sw, sc};
    g.segments = K / 1024 < 1 ? 1 : (K / 1024 > MAX_SEGMENTS ? MAX_SEGMENTS : K / 1024);
    g.segment = ((K + g.segments - 1) / g.segments + BK - 1) / BK * BK;
    g.segments = (K + g.segment - 1) / g.segment;
    g.vec_a = (uintptr_t)A % 16 == 0 && lda % 4 == 0 && sa % 4 == 0;
    g.vec_w = (uintptr_t)W % (4 * sizeof(WT)) == 0 && ldw % 4 == 0 && sw % 4 == 0;
    g.vec_c = (uintptr_t)C % 16 == 0 && ldc % 4 == 0 && sc % 4 == 0;
    if (sizeof(WT) == 4 && batch == 1 && split::takes(N, K, A, W, lda, ldw)) {
        split::Args a = {A, (const float*)W, C, M, N, K, 0, 0, 0, g.vec_c, lda, ldw, ldc};
        return split::product(a, stream);
    }
    // Few rows stream the weights: 32 rows took 73 and 50 us against 119 and 74 in tiles, 48 rows (two passes) 115 and 95 against 121
    // and 78.  (Copies of four values need the alignment; the tiles take everything.)
    if (M <= FEW_ROWS && g.vec_a && g.vec_w) {
        if (M <= 2) return launch_few<WT, 2>(g, batch, stream);
        if (M <= 4) return launch_few<WT, 4>(g, batch, stream);
        if (M <= 8) return launch_few<WT, 8>(g, batch, stream);
        return M <= 16 ? launch_few<WT, 16>(g, batch, stream) : launch_few<WT, 32>(g, batch, stream);
    }
    return dispatch(g, batch, stream);
}

}  // namespace

// A [M,K] row stride lda; W [N,K] row stride ldw (float or bfloat16); C [M,N] row stride ldc.  All of them may be what the kernel before writes.
// `batch` products in one launch: member b reads A + b * sa and W + b * sw and writes C + b * sc.
LLME_API int llme_gemm_nt_f32_batched(const float* A, const void* W, int w_dtype, float* C, int M, int N, int K, long long lda,
                                      long long ldw, long long ldc, int batch, long long sa, long long sw, long long sc,
                                      cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    if (!A || !W || !C || K <= 0) LLME_REFUSE("gemm_f32: null pointer or non-positive K");
    if (batch == 1) sa = sw = sc = 0;                      // (unused)
    // (a batch whose rows lie between those of its other members has a row stride longer than the row)
    if (lda < K || ldw < K || ldc < N) LLME_REFUSE("gemm_f32: a row stride is shorter than the row");
    if ((M + 63) / 64 > 65535 || batch > 65535) LLME_REFUSE("gemm_f32: M = %d or a batch of %d needs more than 65535 grid planes", M, batch);
    if (w_dtype == LLME_F32) return product(A, (const float*)W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
    if (w_dtype == LLME_BF16) return product(A, (const __nv_bfloat16*)W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
    LLME_REFUSE("gemm_f32: unsupported weight dtype %d", w_dtype);
}

LLME_API int llme_gemm_nt_f32(const float* A, const void* W, int w_dtype, float* C, int M, int N, int K,
                              long long lda, long long ldw, long long ldc, cudaStream_t stream) {
    return llme_gemm_nt_f32_batched(A, W, w_dtype, C, M, N, K, lda, ldw, ldc, 1, 0, 0, 0, stream);
}

// 0, or where a bounded wait of the tensor-core form gave up.
LLME_API int llme_gemm_f32_status() { LLME_TAKE_STATUS(split::g_status); }
