// The gated delta rule over portions, 64 tokens at a time on the tensor cores.  Included by delta_rule.cu inside its unnamed namespace;
// heads of 128 rows, columns in whole groups of 32.
//
// The rule over a chunk of tokens, with G(i, j) the product of the decays of tokens j + 1 .. i, G(i) from the chunk's start and S the state
// before it:
//   r_i = b_i (v_i - G(i) S^T k_i),   u = N r,   o_i = G(i) S^T q_i + (B u)_i,   S <- G(63) S + sum_j k_j (G(63, j) u_j)^T,
// N the inverse of the unit lower triangular I + A, A_ij = b_i G(i, j) k_j . k_i, B_ij = G(i, j) k_j . q_i.
//
//   * chunk_prepare_kernel makes what no column of S has a say in, a block per chunk and query/key group: unit vectors, N, B and three
//     numbers a token, by 32-bit multiply-adds.
//   * chunk_walk_kernel walks a request's chunks, a block per (32 columns, head): four products a chunk, [K; Q] S, [N; B] r, K^T u' and
//     [N; B] u, each of 32-bit values split into three bfloat16 pieces (split32.cuh) with sums of at most 64 values in tensor memory.
//     The state stays in 32-bit registers, a row of S a thread.  [K; Q] and [N; B] are first operands in tensor memory; K^T comes from
//     shared memory with its tokens as the summed side; S, r, u and u' are written there as they lie in the threads, 64-byte rows.
//     Eight warps walk, eight split the next chunk's operands, one issues, one copies.
// No quotient of decays is formed.  A chunk at a portion's end is filled up with tokens that change nothing (k = q = 0, b = 0, a = 1).
// A value that is not finite would reach tokens before its own through the zeros of N and B: a block that meets one in u goes on token by token.
// Bound by the chain of the four products of a chunk and the exchanges between them, some 7,000 cycles for 64 tokens, behind a preparation
// whose eleven warps an SM wait for shared memory and at barriers (its path is 32 % busy, the multiply-adds 23 %).  Two portions of 750 tokens, 16 heads of 128 x 128: 91 us, 157 us eight tokens at a
// time (the preparation 41 us, of which 6 beside the walk); four of 375 with 32 heads 181 and 248, one of 2,048 with 32 heads 223 and 413.  Errors
// against 64 bits, of the outputs 1.75e-7 (eight at a time 1.7e-7), of the state 1.2e-7 both.  (The tensor cores cut off what they add instead of
// rounding it: that error has a sign, but goes no further than the 64 values of a sum, about 2^-24 of its largest part a step.)
#pragma once

namespace chunks {

#include "umma.cuh"
#include "split32.cuh"

constexpr int CHUNK = 64, N_ROWS = 128, P_COLS = 32;               // tokens; rows of the state; columns a block takes
constexpr int COEF = 2 * CHUNK * CHUNK + 4 * CHUNK;                // floats per chunk and head: [N; B] as shared memory has it, then b, G and G(63, .) of every token

__device__ __forceinline__ int request_of(const LlmeDeltaArgs& a, int place) { return a.rows ? a.rows[place] : place; }
// Number of the first chunk of the portion at `place` among the rows, distinct for all chunks of a step: floor(first token / 64) + place where
// this form takes all portions (from = 0).  Where it takes those of LONG tokens and more (from = LONG), floor(first token / LONG) stands for the place,
// which the shorter ones would push on: it grows by one at least from one of the others to the next.
__device__ __forceinline__ int first_chunk(const LlmeDeltaArgs& a, int place, int from) {
    const int t = a.cu_q_lens[request_of(a, place)];
    return t / CHUNK + (from > 0 ? t / LONG : place);
}

// where element j of row i of [N; B] lies: two halves of 32 columns, 128-byte rows, their 16-byte pieces swizzled with the row
__device__ __forceinline__ int nb_place(int i, int j) { return (j >> 5) * (2 * CHUNK * 32) + i * 32 + ((((j & 31) >> 2) ^ (i & 7)) << 2) + (j & 3); }

// ----------------------------------------------------------------------------- what no column has a say in
constexpr int PREPARE_THREADS = 256, ROW = N_ROWS + 4, TRI = CHUNK + 4;
struct PrepareShared {
    union {
        float kq[2][CHUNK][ROW];                                   // unit keys and queries
        float tri[6][CHUNK][TRI];                                  // k . k, k . q, A of two heads (N in the end), B of two heads
    };
    float beta[2][CHUNK], keep[2][CHUNK];
};

__global__ void __launch_bounds__(PREPARE_THREADS, 2) chunk_prepare_kernel(LlmeDeltaArgs a, int from) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PrepareShared& sm = *reinterpret_cast<PrepareShared*>(smem_raw);
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, id = blockIdx.x, g = blockIdx.y;
    int place = 0, hi = a.n_rows;                                  // the last portion whose first chunk is not behind `id`
    while (hi - place > 1) {
        const int mid = (place + hi) >> 1;
        if (first_chunk(a, mid, from) <= id) place = mid; else hi = mid;
    }
    const int r = request_of(a, place), first = a.cu_q_lens[r], at = CHUNK * (id - first_chunk(a, place, from)), len = a.cu_q_lens[r + 1] - first;
    if (at < 0 || at >= len || len < from) return;                 // a number no chunk has, or a portion of the other form
    const int t0 = first + at, count = min(CHUNK, len - at);
    const int rep = a.heads / a.qk_groups, x = tid >> 7, t = tid & 127, j = tid & 63;
    const bool lower = !(tid & 64);
    float2 gate = make_float2(0.0f, 0.0f);                         // of the next two heads, on their way while other work goes on
    auto load_gate = [&](int head) {
        if (lower && head < rep && j < count) {
            const size_t at = (size_t)(t0 + j) * a.ld_gates + g * rep + head;
            gate = make_float2(a.write[at], a.forget[at]);
        }
    };
    load_gate(x);
    // unit vectors: a warp takes eight tokens, a lane four values of each
    {
        float4 k[8], q[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = warp * 8 + i;
            k[i] = q[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (t < count) {
                k[i] = *reinterpret_cast<const float4*>(a.k + (size_t)(t0 + t) * a.ldk + (size_t)g * N_ROWS + 4 * lane);
                q[i] = *reinterpret_cast<const float4*>(a.q + (size_t)(t0 + t) * a.ldq + (size_t)g * N_ROWS + 4 * lane);
            }
        }
        // the sixteen sums of squares at once: lanes exchange halves of what they hold until every pair of lanes has one
        float ss[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            ss[i] = fmaf(k[i].x, k[i].x, fmaf(k[i].y, k[i].y, fmaf(k[i].z, k[i].z, k[i].w * k[i].w)));
            ss[8 + i] = fmaf(q[i].x, q[i].x, fmaf(q[i].y, q[i].y, fmaf(q[i].z, q[i].z, q[i].w * q[i].w)));
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const bool up = lane & (2 * o);
#pragma unroll
            for (int i = 0; i < o; ++i) ss[i] = (up ? ss[i + o] : ss[i]) + __shfl_xor_sync(0xffffffffu, up ? ss[i] : ss[i + o], 2 * o);
        }
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);           // lane 2 i (and the next): sum i
        const float inverse = (lane < 16 ? 1.0f : a.q_scale) / sqrtf(ss[0] + a.unit_eps);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = warp * 8 + i;
            const float ik = __shfl_sync(0xffffffffu, inverse, 2 * i), iq = __shfl_sync(0xffffffffu, inverse, 16 + 2 * i);
            k[i] = make_float4(k[i].x * ik, k[i].y * ik, k[i].z * ik, k[i].w * ik);
            q[i] = make_float4(q[i].x * iq, q[i].y * iq, q[i].z * iq, q[i].w * iq);
            *reinterpret_cast<float4*>(&sm.kq[0][t][4 * lane]) = k[i];
            *reinterpret_cast<float4*>(&sm.kq[1][t][4 * lane]) = q[i];
            if (t < count) {
                float* u = a.unit + ((size_t)(t0 + t) * 2 * a.qk_groups + g) * N_ROWS + 4 * lane;
                *reinterpret_cast<float4*>(u) = q[i];
                *reinterpret_cast<float4*>(u + (size_t)a.qk_groups * N_ROWS) = k[i];
            }
        }
    }
    __syncthreads();
    // k_i . k_j and q_i . k_j for rows 4 ty .. + 3 and columns tx + 16 c; a warp holds eight rows and leaves out what lies behind them
    const int ty = tid >> 4, tx = tid & 15, most = warp >> 1;      // (columns 16 c and on are needed while 16 c <= 8 warp + 7)
    float kk[4][4], qk[4][4];
    auto products = [&](const float (*rows)[ROW], float (&sum)[4][4]) {
        // Sums of sixteen products (two of eight side by side), added up with what each addition lost carried along: errors of these sums are
        // met by every token behind, and one chain of 128 made the whole rule's error 1.4 times as large.
        float lost[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) sum[i][c] = lost[i][c] = 0.0f;
#pragma unroll 1
        for (int e0 = 0; e0 < N_ROWS; e0 += 16) {
            unsigned long long part[4][4];
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
                ulonglong2 mine[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) mine[i] = *reinterpret_cast<const ulonglong2*>(&rows[4 * ty + i][e0 + e]);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (c > most) break;
                    const ulonglong2 kj = *reinterpret_cast<const ulonglong2*>(&sm.kq[0][tx + 16 * c][e0 + e]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (e == 0) asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(part[i][c]) : "l"(mine[i].x), "l"(kj.x));
                        else asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(part[i][c]) : "l"(mine[i].x), "l"(kj.x));
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(part[i][c]) : "l"(mine[i].y), "l"(kj.y));
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (c > most) break;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float y = (__uint_as_float((unsigned)part[i][c]) + __uint_as_float((unsigned)(part[i][c] >> 32))) - lost[i][c], next = sum[i][c] + y;
                    lost[i][c] = (next - sum[i][c]) - y;
                    sum[i][c] = next;
                }
            }
        }
    };
    products(sm.kq[0], kk);
    products(sm.kq[1], qk);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sm.tri[0][4 * ty + i][tx + 16 * c] = kk[i][c];
            sm.tri[1][4 * ty + i][tx + 16 * c] = qk[i][c];
        }
    // two heads at a time, 128 threads each: thread j of the first 64 (`lower`) forms rows 0 .. 31 of column j of A and B, thread j of the others
    // rows 32 .. 63 and token j's numbers; then all of them N
    for (int x0 = 0; x0 < rep; x0 += 2) {
        const bool here = x0 + x < rep;
        const int h = g * rep + x0 + x;
        float (*A)[TRI] = sm.tri[2 + x], (*B)[TRI] = sm.tri[4 + x];
        if (here && lower) {
            float beta = 0.0f, keep = 1.0f;
            if (j < count) {
                beta = write_strength(gate.x);
                keep = decay_of(gate.y + a.dt_bias[h], a.a_log[h]);
            }
            sm.beta[x][j] = beta;
            sm.keep[x][j] = keep;
        }
        load_gate(x0 + 2 + x);
        __syncthreads();
        float* coef = a.coef + ((size_t)id * a.heads + h) * COEF;
        if (here) {
            // (64 bits: rounded to 32 once, in A and B; products of up to 64 decays would have a rounding each)
            double G = 1.0, from_start = 1.0;
            const int first_row = lower ? 0 : CHUNK / 2;
            if (!lower)
#pragma unroll 8
                for (int i = 0; i < CHUNK / 2; ++i) {
                    const double w = sm.keep[x][i];
                    if (i > j) G *= w;
                    if (i <= j) from_start *= w;
                }
#pragma unroll
            for (int i0 = 0; i0 < CHUNK / 2; i0 += 4) {
                const float4 w4 = *reinterpret_cast<const float4*>(&sm.keep[x][first_row + i0]), b4 = *reinterpret_cast<const float4*>(&sm.beta[x][first_row + i0]);
                const float w[4] = {w4.x, w4.y, w4.z, w4.w}, beta[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = first_row + i0 + e;
                    if (i > j) G *= (double)w[e];                  // G(i, j)
                    else from_start *= (double)w[e];
                    A[i][j] = i > j ? (float)(G * ((double)beta[e] * (double)sm.tri[0][i][j])) : 0.0f;
                    B[i][j] = i >= j ? (float)(G * (double)sm.tri[1][i][j]) : 0.0f;
                }
            }
            if (!lower) *reinterpret_cast<float4*>(coef + 2 * CHUNK * CHUNK + 4 * j) = make_float4(sm.beta[x][j], (float)from_start, (float)G, 0.0f);
        }
        __syncthreads();
        // N in place of A (strictly below the diagonal): blocks of 16 by substitution, a column a thread, then [N1 0; -N2 A N1 N2] for blocks of 32 and of 64
        if (here && lower) {
            const int b0 = j & ~15, jj = j & 15;
            float N[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
                for (int m = 0; m < i; ++m) (m & 1 ? s1 : s0) = fmaf(A[b0 + i][b0 + m], N[m], m & 1 ? s1 : s0);
                N[i] = (i == jj ? 1.0f : 0.0f) - (s0 + s1);        // (exactly 0 above the diagonal)
            }
            __syncwarp();                                          // (a block's sixteen columns are one half of a warp)
#pragma unroll
            for (int i = 0; i < 16; ++i) A[b0 + i][j] = N[i];
        }
        __syncthreads();
        auto join = [&](auto block) {
            constexpr int size = decltype(block)::value;
            // pairs of blocks p: T = A21 N11 (rows r .. of the pair's lower left block), then N21 = -N22 T
            constexpr int pairs = CHUNK / (2 * size), per_pair = 128 / pairs, outs = size * size / per_pair;
            const int p = t / per_pair, u = t % per_pair;
            const int b0 = p * 2 * size, row = b0 + size + u / (size / 4) * (4 * outs / 16), c0 = b0 + (u % (size / 4)) * 4;
            float T[2][4];                                         // outs / 4 rows of four columns
#pragma unroll 1
            for (int turn = 0; turn < 2; ++turn) {
                if (here)
                {
                    // turn 0: A21 [row, m] N11 [m, c]; turn 1: N22 [row, m] T [m, c]
                    const int at = turn == 0 ? b0 : b0 + size;
#pragma unroll
                    for (int i = 0; i < outs / 4; ++i) T[i][0] = T[i][1] = T[i][2] = T[i][3] = 0.0f;
#pragma unroll 2
                    for (int m = 0; m < size; m += 4) {
                        float4 l[outs / 4];
#pragma unroll
                        for (int i = 0; i < outs / 4; ++i) l[i] = *reinterpret_cast<const float4*>(&A[row + i][at + m]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float4 v = *reinterpret_cast<const float4*>(&A[at + m + e][c0]);
#pragma unroll
                            for (int i = 0; i < outs / 4; ++i) {
                                const float le = e == 0 ? l[i].x : e == 1 ? l[i].y : e == 2 ? l[i].z : l[i].w;
                                T[i][0] = fmaf(le, v.x, T[i][0]); T[i][1] = fmaf(le, v.y, T[i][1]); T[i][2] = fmaf(le, v.z, T[i][2]); T[i][3] = fmaf(le, v.w, T[i][3]);
                            }
                        }
                    }
                }
                __syncthreads();
                if (here)
#pragma unroll
                    for (int i = 0; i < outs / 4; ++i)
                        *reinterpret_cast<float4*>(&A[row + i][c0]) = turn == 0 ? make_float4(T[i][0], T[i][1], T[i][2], T[i][3]) : make_float4(-T[i][0], -T[i][1], -T[i][2], -T[i][3]);
                __syncthreads();
            }
        };
        join(std::integral_constant<int, 16>{});
        join(std::integral_constant<int, 32>{});
        if (here)
            for (int i = t; i < CHUNK * (CHUNK / 4); i += 128) {
                const int row = i / (CHUNK / 4), c = (i % (CHUNK / 4)) * 4;
                *reinterpret_cast<float4*>(coef + nb_place(row, c)) = *reinterpret_cast<const float4*>(&A[row][c]);
                *reinterpret_cast<float4*>(coef + nb_place(CHUNK + row, c)) = *reinterpret_cast<const float4*>(&B[row][c]);
            }
        __syncthreads();
    }
}

// ----------------------------------------------------------------------------- the walk
constexpr int KQ_RAW = 2 * CHUNK * N_ROWS * 4, NB_RAW = 2 * CHUNK * CHUNK * 4, KT_PLANE = CHUNK * N_ROWS * 2, S_PLANE = N_ROWS * P_COLS * 2, U_PLANE = CHUNK * P_COLS * 2;
// tensor memory: [K; Q], [N; B], then the products: [K; Q] S, N r, B u, K^T u'
constexpr int DS_SUMS = 2, DU_SUMS = 2, DO_SUMS = 2;               // sums of 64, 32 and 32 values, added up in registers
constexpr unsigned KQ_COL = 0, NB_COL = PIECES * N_ROWS / 2, DS_COL = NB_COL + PIECES * CHUNK / 2, DU_COL = DS_COL + DS_SUMS * P_COLS, DO_COL = DU_COL + DU_SUMS * P_COLS,
                   DN_COL = DO_COL + DO_SUMS * P_COLS;
constexpr int WALKERS = 8, SPLITTERS = 8, WALK_ISSUER = WALKERS + SPLITTERS, WALK_THREADS = (WALK_ISSUER + 2) * 32, MINE = P_COLS / 2;     // MINE: columns a walking thread has

struct WalkBarriers {
    unsigned long long raw_full, raw_empty;                        // copied operands of a chunk
    unsigned long long kq_ready, nb_ready, kt_ready, s_ready, r_ready, up_ready, u_ready;      // split operands
    unsigned long long ds_done, du_done, dn_done, do_done;         // products: [K; Q] S, N r, K^T u', B u
    unsigned tmem_base;
    int abort_flag, alone_flag;                                    // (the second of waits that no other role ends)
    int plain;                                                     // a value that is not finite was met: the rest goes token by token
    float part[2][WALKERS][MINE];
};

// 64-byte rows of 32 values, the other side of the product: eight rows of the summed side are a group of 512 bytes (64-byte swizzle)
__device__ __forceinline__ unsigned long long desc_rows64(const void* tile) {
    return (unsigned long long)((smem_u32(tile) & 0x3FFFFu) >> 4) | (unsigned long long)1 << 16 | (unsigned long long)(512 >> 4) << 32 |
           (unsigned long long)1 << 46 | (unsigned long long)4 << 61;
}
// two halves of 64 values in 128-byte rows, CHUNK rows of the summed side each (128-byte swizzle)
__device__ __forceinline__ unsigned long long desc_rows128(const void* tile) {
    return (unsigned long long)((smem_u32(tile) & 0x3FFFFu) >> 4) | (unsigned long long)((CHUNK * 128) >> 4) << 16 | (unsigned long long)(1024 >> 4) << 32 |
           (unsigned long long)1 << 46 | (unsigned long long)2 << 61;
}
// MINE values of a thread's row, from column `col` on, into 64-byte rows, piece p at tile + p * plane
__device__ __forceinline__ void store_split(const float (&x)[MINE], unsigned char* tile, int row, int col, int plane) {
#pragma unroll
    for (int i = 0; i < MINE / 8; ++i)
        split8_to_smem<true>(make_float4(x[8 * i], x[8 * i + 1], x[8 * i + 2], x[8 * i + 3]), make_float4(x[8 * i + 4], x[8 * i + 5], x[8 * i + 6], x[8 * i + 7]),
                       tile + row * 64 + (((col / 8 + i) ^ ((row >> 1) & 3)) << 4), plane);
}
__device__ __forceinline__ void tmem_load16(unsigned addr, unsigned (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(addr));
}
// MINE columns of a product, held in SUMS parts
template <int SUMS>
__device__ __forceinline__ void load_product(unsigned addr, float (&x)[MINE]) {
    static_assert(MINE == 16 && SUMS <= 2, "one load a part");
    unsigned v[SUMS][16];
#pragma unroll
    for (int i = 0; i < SUMS; ++i) tmem_load16(addr + (unsigned)(i * P_COLS), v[i]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < MINE; ++i) x[i] = SUMS > 1 ? __uint_as_float(v[0][i]) + __uint_as_float(v[SUMS - 1][i]) : __uint_as_float(v[0][i]);
}

constexpr size_t WALK_SMEM = 1024 + PIECES * KT_PLANE + PIECES * S_PLANE + 2 * PIECES * U_PLANE + KQ_RAW + NB_RAW + sizeof(WalkBarriers);

__global__ void __launch_bounds__(WALK_THREADS, 1) chunk_walk_kernel(const __grid_constant__ CUtensorMap map_unit, LlmeDeltaArgs a, int from) {
    static_assert(DN_COL + P_COLS <= 512 && WALK_SMEM <= 232448, "sizes");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* kq_raw = smem;                                  // keys, then queries: four times [64 tokens][32 values] each
    unsigned char* nb_raw = kq_raw + KQ_RAW;                       // [N; B]: two times [128 rows][32 values]
    unsigned char* kt = nb_raw + NB_RAW;                           // pieces of K: two halves of [64 tokens][64 rows of the state]
    unsigned char* s_tile = kt + PIECES * KT_PLANE;                // pieces of S: [128 rows][32 columns]
    unsigned char* r_tile = s_tile + PIECES * S_PLANE;             // pieces of r, then of u': [64 tokens][32 columns]
    unsigned char* u_tile = r_tile + PIECES * U_PLANE;             // pieces of u
    WalkBarriers* bar = reinterpret_cast<WalkBarriers*>(u_tile + PIECES * U_PLANE);
    volatile int* abort_flag = &bar->abort_flag;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&bar->raw_full, 1); mbar_init(&bar->raw_empty, SPLITTERS);
        mbar_init(&bar->kq_ready, SPLITTERS); mbar_init(&bar->nb_ready, SPLITTERS); mbar_init(&bar->kt_ready, SPLITTERS);
        mbar_init(&bar->s_ready, WALKERS); mbar_init(&bar->r_ready, WALKERS / 2); mbar_init(&bar->up_ready, WALKERS / 2); mbar_init(&bar->u_ready, WALKERS);
        mbar_init(&bar->ds_done, 1); mbar_init(&bar->du_done, 1); mbar_init(&bar->dn_done, 1); mbar_init(&bar->do_done, 1);
        bar->abort_flag = bar->alone_flag = bar->plain = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WALK_ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bar->tmem_base)), "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_wait();
    const int p0 = blockIdx.x * P_COLS, h = blockIdx.y, r = request_of(a, blockIdx.z), g = h / (a.heads / a.qk_groups);
    const int first = a.cu_q_lens[r], len = a.cu_q_lens[r + 1] - first, n_chunks = (len + CHUNK - 1) / CHUNK, id0 = first_chunk(a, blockIdx.z, from);
    if (len <= 0 || len < from) {                                  // an empty portion, or one of the other form: neither outputs nor a state to write
        if (warp == WALK_ISSUER) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(bar->tmem_base), "r"(512u));
        return;
    }
    auto coef_of = [&](int c) { return a.coef + ((size_t)(id0 + c) * a.heads + h) * COEF; };
    const unsigned tmem = bar->tmem_base;
    auto after = [] { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); };
    auto before = [] { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); };
    auto publish = [] { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); };     // what the instructions read through the async proxy

    if (warp < WALKERS) {
        // ------------------------------------------------------------------ the walk: row `row` of S, token `tok` of the chunk, columns col .. col + MINE - 1
        const int row = tid & 127, tok = row & 63, col = (warp >> 2) * MINE;
        const bool keys = row < CHUNK;                             // lanes of K (and of N: r and u); the others of Q (and of B: the outputs)
        const unsigned mine = tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)col;
        float* st = a.state + (size_t)a.state_slots[r] * a.state_stride + ((size_t)h * a.p + p0 + col) * N_ROWS + row;
        float S[MINE], o[MINE], weight = 0.0f;
#pragma unroll
        for (int i = 0; i < MINE; ++i) S[i] = st[(size_t)i * N_ROWS];
        auto write_out = [&](int c) {                              // outputs of chunk c: G S^T q + B u
            float d[MINE];
            after();
            load_product<DO_SUMS>(mine + DO_COL, d);
            if (c * CHUNK + tok < len) {
                float* out = a.out + (size_t)(first + c * CHUNK + tok) * a.ldo + (size_t)h * a.p + p0 + col;
#pragma unroll
                for (int i = 0; i < MINE; i += 4) *reinterpret_cast<float4*>(out + i) = make_float4(fmaf(weight, o[i], d[i]), fmaf(weight, o[i + 1], d[i + 1]), fmaf(weight, o[i + 2], d[i + 2]), fmaf(weight, o[i + 3], d[i + 3]));
            }
            before();
        };
        auto split = [&](const float (&x)[MINE], unsigned char* tile, int at, int plane, unsigned long long* ready) {
            store_split(x, tile, at, col, plane);
            publish();
            before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready);
        };
        bool ok = true;
        int c = 0;
        for (; c < n_chunks && ok; ++c) {
            const unsigned now = (unsigned)c & 1;
            const bool real = c * CHUNK + tok < len;
            split(S, s_tile, row, S_PLANE, &bar->s_ready);
            const float4 num = *reinterpret_cast<const float4*>(coef_of(c) + 2 * CHUNK * CHUNK + 4 * tok);       // b, G, G(63, .)
            const float total = coef_of(c)[2 * CHUNK * CHUNK + 4 * (CHUNK - 1) + 1];
            float4 v[MINE / 4];
            if (keys)
#pragma unroll
                for (int i = 0; i < MINE / 4; ++i)
                    v[i] = real ? *reinterpret_cast<const float4*>(a.v + (size_t)(first + c * CHUNK + tok) * a.ldv + (size_t)h * a.p + p0 + col + 4 * i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            else {
                if (c > 0) {
                    if (!(ok = mbar_wait(&bar->do_done, now ^ 1, &bar->alone_flag, 1))) break;
                    write_out(c - 1);
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive(&bar->u_ready);         // (the outputs of the chunk before have been read)
            }
            if (!(ok = mbar_wait(&bar->ds_done, now, abort_flag, 2))) break;
            float d[MINE];
            after();
            load_product<DS_SUMS>(mine + DS_COL, d);
            if (keys) {
                const float* vv = reinterpret_cast<const float*>(v);
#pragma unroll
                for (int i = 0; i < MINE; ++i) d[i] = real ? num.x * fmaf(-num.y, d[i], vv[i]) : 0.0f;
                split(d, r_tile, tok, U_PLANE, &bar->r_ready);
                if (!(ok = mbar_wait(&bar->du_done, now, abort_flag, 3))) break;
                after();
                load_product<DU_SUMS>(mine + DU_COL, d);
                float up[MINE];
#pragma unroll
                for (int i = 0; i < MINE; ++i) up[i] = num.z * d[i];
                // Zeros of N, B and K^T would carry a value that is not finite to tokens before it: the chunk and what follows go token by token instead
                float off = 0.0f;
#pragma unroll
                for (int i = 0; i < MINE; ++i) off = fmaf(d[i], 0.0f, off);
                if (__any_sync(0xffffffffu, off != 0.0f)) {
                    bar->plain = 1;
                    *abort_flag = -1;
                    ok = false;
                    break;
                }
                split(up, r_tile, tok, U_PLANE, &bar->up_ready);
                split(d, u_tile, tok, U_PLANE, &bar->u_ready);
            } else {
#pragma unroll
                for (int i = 0; i < MINE; ++i) o[i] = d[i];
                weight = num.y;
                before();
            }
            if (!(ok = mbar_wait(&bar->dn_done, now, abort_flag, 4))) break;
            after();
            load_product<1>(mine + DN_COL, d);
            before();
#pragma unroll
            for (int i = 0; i < MINE; ++i) S[i] = fmaf(total, S[i], d[i]);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(WALKERS * 32) : "memory");
        if (*(volatile int*)&bar->plain) {                         // (no warp has gone past this chunk's S: that needs u of all of it)
            const float* unit = a.unit + (size_t)g * N_ROWS + row;
            const int group = warp & ~3;                           // the four warps of these columns
            auto add_rows = [&](float (&x)[MINE], float (&part)[WALKERS][MINE]) {
#pragma unroll
                for (int i = 0; i < MINE; ++i) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) x[i] += __shfl_xor_sync(0xffffffffu, x[i], o);
                    if (lane == 0) part[warp][i] = x[i];
                }
                asm volatile("bar.sync 1, %0;" ::"n"(WALKERS * 32) : "memory");
            };
            for (int t = c * CHUNK; t < len; ++t) {
                const size_t at = (size_t)(first + t);
                const float q = unit[at * 2 * a.qk_groups * N_ROWS], k = unit[(at * 2 + 1) * a.qk_groups * N_ROWS];
                const float beta = write_strength(a.write[at * a.ld_gates + h]), keep = decay_of(a.forget[at * a.ld_gates + h] + a.dt_bias[h], a.a_log[h]);
                float x[MINE];
#pragma unroll
                for (int i = 0; i < MINE; ++i) x[i] = (S[i] *= keep) * k;
                add_rows(x, bar->part[0]);
#pragma unroll
                for (int i = 0; i < MINE; ++i) {
                    const float have = (bar->part[0][group][i] + bar->part[0][group + 1][i]) + (bar->part[0][group + 2][i] + bar->part[0][group + 3][i]);
                    S[i] = fmaf(k, beta * (a.v[at * a.ldv + (size_t)h * a.p + p0 + col + i] - have), S[i]);
                    x[i] = S[i] * q;
                }
                add_rows(x, bar->part[1]);
                if (tid < P_COLS) {
                    const int w = tid / MINE * 4, i = tid % MINE;
                    a.out[at * a.ldo + (size_t)h * a.p + p0 + tid] = (bar->part[1][w][i] + bar->part[1][w + 1][i]) + (bar->part[1][w + 2][i] + bar->part[1][w + 3][i]);
                }
            }
#pragma unroll
            for (int i = 0; i < MINE; ++i) st[(size_t)i * N_ROWS] = S[i];
        }
        if (ok && !keys && mbar_wait(&bar->do_done, (unsigned)(n_chunks - 1) & 1, abort_flag, 5)) write_out(n_chunks - 1);
        if (ok)
#pragma unroll
            for (int i = 0; i < MINE; ++i) st[(size_t)i * N_ROWS] = S[i];
    } else if (warp < WALK_ISSUER) {
        // ------------------------------------------------------------------ the next chunk's operands
        const int u = tid - WALKERS * 32, t = u & 127, half = u >> 7;      // row of [K; Q] and of [N; B], half of its values
        const unsigned mine = tmem + ((unsigned)((warp & 3) * 32) << 16);
        for (int c = 0; c < n_chunks; ++c) {
            const unsigned now = (unsigned)c & 1;
            const int count = min(CHUNK, len - c * CHUNK);
            if (!mbar_wait(&bar->raw_full, now, abort_flag, 6) || !mbar_wait(&bar->ds_done, now ^ 1, abort_flag, 7)) break;
            after();
            const bool real = (t & 63) < count;
#pragma unroll
            for (int qq = 0; qq < N_ROWS / 32; ++qq) {
                const int q = half * (N_ROWS / 32) + qq;
                float4 x[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    x[i] = real ? *reinterpret_cast<const float4*>(kq_raw + (t >> 6) * (KQ_RAW / 2) + (q >> 1) * (CHUNK * 128) + (t & 63) * 128 + ((((q & 1) * 4 + i) ^ (t & 7)) << 4))
                                : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                split16_to_tmem<false>(x, mine + KQ_COL + (unsigned)(q * 8), N_ROWS / 2);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->kq_ready);
            if (!mbar_wait(&bar->do_done, now ^ 1, abort_flag, 9)) break;
            after();
#pragma unroll
            for (int qq = 0; qq < CHUNK / 32; ++qq) {
                const int q = half * (CHUNK / 32) + qq;
                float4 x[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(nb_raw + (q >> 1) * (NB_RAW / 2) + t * 128 + ((((q & 1) * 4 + i) ^ (t & 7)) << 4));
                split16_to_tmem<false>(x, mine + NB_COL + (unsigned)(q * 8), CHUNK / 2);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar->nb_ready);
            // (all products of the chunk before are done: K's tiles are free)
#pragma unroll 2
            for (int j = 0; j < CHUNK * N_ROWS / 8 / (SPLITTERS * 32); ++j) {
                const int i = u + SPLITTERS * 32 * j, tokn = (i & 7) + 8 * (i >> 7), q = (i >> 3) & 15;
                float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
                if (tokn < count) {
                    const unsigned char* src = kq_raw + (q >> 2) * (CHUNK * 128) + tokn * 128;
                    lo = *reinterpret_cast<const float4*>(src + (((2 * (q & 3)) ^ (tokn & 7)) << 4));
                    hi = *reinterpret_cast<const float4*>(src + (((2 * (q & 3) + 1) ^ (tokn & 7)) << 4));
                }
                split8_to_smem<false>(lo, hi, kt + (q >> 3) * (CHUNK * 128) + tokn * 128 + (((q & 7) ^ (tokn & 7)) << 4), KT_PLANE);
            }
            publish();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bar->kt_ready);
                mbar_arrive(&bar->raw_empty);
            }
        }
    } else if (warp == WALK_ISSUER) {
        // ------------------------------------------------------------------ the products
        constexpr unsigned id_rows = umma_idesc(BM, P_COLS) | (1u << 16);              // second operand by rows of the summed side
        constexpr unsigned id_both = id_rows | (1u << 15);                             // the first one too
        const unsigned long long s_desc = desc_rows64(s_tile), r_desc = desc_rows64(r_tile), u_desc = desc_rows64(u_tile), k_desc = desc_rows128(kt);
        auto from_tmem = [&](unsigned d, unsigned first_col, int step, unsigned long long b, int plane, int steps, int sums) {
#pragma unroll
            for (int part = 0; part < sums; ++part)
#pragma unroll
                for (int i = 0; i < PAIRS; ++i)
#pragma unroll
                    for (int k = part * steps / sums; k < (part + 1) * steps / sums; ++k)
                        umma_from_tmem(tmem + d + (unsigned)(part * P_COLS), tmem + first_col + (unsigned)(SecondUp::a(i) * step + k * 8),
                                       b + (unsigned long long)(SecondUp::b(i) * (plane >> 4) + k * 64), id_rows, i > 0 || k > part * steps / sums,
                                       k == part * steps / sums && SecondUp::steps_down(i));
        };
        for (int c = 0; c < n_chunks; ++c) {
            const unsigned now = (unsigned)c & 1;
            if (!mbar_wait(&bar->s_ready, now, abort_flag, 10) || !mbar_wait(&bar->kq_ready, now, abort_flag, 11)) break;
            after();
            if (elect_one()) {
                from_tmem(DS_COL, KQ_COL, N_ROWS / 2, s_desc, S_PLANE, N_ROWS / UMMA_K, DS_SUMS);
                umma_commit(&bar->ds_done);
            }
            __syncwarp();
            if (!mbar_wait(&bar->r_ready, now, abort_flag, 12) || !mbar_wait(&bar->nb_ready, now, abort_flag, 13)) break;
            after();
            if (elect_one()) {
                from_tmem(DU_COL, NB_COL, CHUNK / 2, r_desc, U_PLANE, CHUNK / UMMA_K, DU_SUMS);
                umma_commit(&bar->du_done);
            }
            __syncwarp();
            if (!mbar_wait(&bar->up_ready, now, abort_flag, 14) || !mbar_wait(&bar->kt_ready, now, abort_flag, 15)) break;
            after();
            if (elect_one()) {
#pragma unroll
                for (int i = 0; i < PAIRS; ++i)
#pragma unroll
                    for (int k = 0; k < CHUNK / UMMA_K; ++k)
                        umma_from_smem(tmem + DN_COL, k_desc + (unsigned long long)(SecondUp::a(i) * (KT_PLANE >> 4) + k * 128), r_desc + (unsigned long long)(SecondUp::b(i) * (U_PLANE >> 4) + k * 64),
                                  id_both, i > 0 || k > 0, k == 0 && SecondUp::steps_down(i));
                umma_commit(&bar->dn_done);
            }
            __syncwarp();
            if (!mbar_wait(&bar->u_ready, now, abort_flag, 16)) break;
            after();
            if (elect_one()) {
                from_tmem(DO_COL, NB_COL, CHUNK / 2, u_desc, U_PLANE, CHUNK / UMMA_K, DO_SUMS);
                umma_commit(&bar->do_done);
            }
            __syncwarp();
        }
    } else {
        // ------------------------------------------------------------------ copies (of rows behind the portion too: what they hold does not count)
        int c = 0;
        for (; c < n_chunks; ++c) {
            if (!mbar_wait(&bar->raw_empty, ((unsigned)c & 1) ^ 1, abort_flag, 17) || *abort_flag) break;
            if (elect_one()) {
                mbar_expect_tx(&bar->raw_full, KQ_RAW + NB_RAW);
#pragma unroll
                for (int i = 0; i < N_ROWS / 32; ++i) {
                    tma_load_2d(kq_raw + i * (CHUNK * 128), &map_unit, (a.qk_groups + g) * N_ROWS + 32 * i, first + c * CHUNK, &bar->raw_full);
                    tma_load_2d(kq_raw + KQ_RAW / 2 + i * (CHUNK * 128), &map_unit, g * N_ROWS + 32 * i, first + c * CHUNK, &bar->raw_full);
                }
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(nb_raw)), "l"(coef_of(c)), "r"(NB_RAW), "r"(smem_u32(&bar->raw_full)) : "memory");
            }
            __syncwarp();
        }
        if (c > 0)                                                 // the copies that may still be in flight land first, also where another role gave up
            for (unsigned i = 0; i < WAIT_LIMIT && !mbar_try_wait(&bar->raw_full, (unsigned)(c - 1) & 1); ++i) {}
    }
    __syncwarp();
    before();
    __syncthreads();
    if (warp == WALK_ISSUER) {
        after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
    }
}

// Whether portions can go 64 tokens at a time: what the forms above need of sizes and alignment, and a workspace that holds the chunks of
// portions of LONG tokens or more.  LONG lies where the forms meet for a portion by itself; eight and 64 at a time (us): 200 tokens of 16 heads 40 and
// 44, 256 46 and 45, 300 52 and 48, 1,500 224 and 138; 32 heads 256 58 and 46, 300 68 and 51.  (Several shorter ones side by side would be faster
// here, four of 192 58 against 68, but what stands beside a portion has no say.)
int most_chunks(const LlmeDeltaArgs& a) { return a.tokens / CHUNK + a.tokens / LONG + 1; }
bool takes(const LlmeDeltaArgs& a) {
    const uintptr_t all = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.out | (uintptr_t)a.unit | (uintptr_t)a.coef;
    return a.n == N_ROWS && a.p % P_COLS == 0 && all % 16 == 0 && (a.ldq | a.ldk | a.ldv | a.ldo) % 4 == 0 && a.tokens >= LONG &&
           (long long)most_chunks(a) * a.heads * COEF <= a.coef_floats && a.qk_groups <= 65535;
}

// The portions of `from` = LONG tokens or more; 0: all, of which there are no more than a.tokens / LONG.
int launch(const LlmeDeltaArgs& a, int from, cudaStream_t s) {
    static LlmeGrants prepare_grants, walk_grants;
    if (llme_grant_smem(prepare_grants, chunk_prepare_kernel, sizeof(PrepareShared)) != cudaSuccess || llme_grant_smem(walk_grants, chunk_walk_kernel, WALK_SMEM) != cudaSuccess)
        LLME_REFUSE("delta_rule: %zu bytes of shared memory are not available", WALK_SMEM);
    CUtensorMap unit;
    if (int rc = make_map(&unit, a.unit, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.tokens, 2LL * a.qk_groups * N_ROWS, 2LL * a.qk_groups * N_ROWS, CHUNK, 32)) return rc;
    llme_launch(chunk_prepare_kernel, dim3(from > 0 ? most_chunks(a) : a.tokens / CHUNK + a.n_rows + 1, a.qk_groups), dim3(PREPARE_THREADS), sizeof(PrepareShared), s, a, from);
    llme_launch(chunk_walk_kernel, dim3(a.p / P_COLS, a.heads, a.n_rows), dim3(WALK_THREADS), WALK_SMEM, s, unit, a, from);
    if (a.launches) *a.launches += 2;
    LLME_LAUNCH_STATUS();
}

}  // namespace chunks
