// A 32-bit value as the sum of three bfloat16 values, for tensor cores that take no 32-bit operands: 24 significant bits are 8 + 8 + 8,
// each piece is what is left rounded to nearest.  x w is then formed from the six products of pieces that reach into 32 bits; what is left out,
// x_2 w_3 + x_3 w_2 + x_3 w_3, is below 2^-25 of |x w|.
// Pieces taken `up` stand 2^8 (the second) and 2^16 (the third) times too high.  So none of a value from 2^-126 on is below bfloat16's smallest
// number, and the three are exact; as they are, the third falls short from 2^-110 on (9e-6 of a product is lost at 2^-118, 4e-2 at 2^-130).  Products
// are added from the highest level down, and where a lower one begins the instruction takes the sum so far times 2^-8.  (A value below 2^-126 has
// its first digits in a later piece, and what is left out grows with that: 3e-7 of a product at 2^-130, 2e-4 at 2^-140.)
// Included behind umma.cuh, inside the including file's namespace.
#pragma once

constexpr int PIECES = 3, PAIRS = 6;
// (piece of the first operand, piece of the second) of the products, in their order: where both operands' pieces are taken up, the least first ...
struct BothUp {
    static __device__ constexpr int a(int pair) { constexpr int of[PAIRS] = {2, 0, 1, 1, 0, 0}; return of[pair]; }
    static __device__ constexpr int b(int pair) { constexpr int of[PAIRS] = {0, 2, 1, 0, 1, 0}; return of[pair]; }
    static __device__ constexpr bool steps_down(int pair) { return pair == 3 || pair == 5; }
};
// ... and where the second operand's are
struct SecondUp {
    static __device__ constexpr int a(int pair) { constexpr int of[PAIRS] = {0, 1, 0, 2, 1, 0}; return of[pair]; }
    static __device__ constexpr int b(int pair) { constexpr int of[PAIRS] = {2, 1, 1, 0, 0, 0}; return of[pair]; }
    static __device__ constexpr bool steps_down(int pair) { return pair == 1 || pair == 3; }
};

// Two neighbouring values: the next piece of both, packed, which they lose unless it is the last; UP: what is left is taken 2^8 times.
template <bool UP>
__device__ __forceinline__ unsigned take_piece(float& lo, float& hi, bool last) {
    unsigned p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(hi), "f"(lo));
    if (!last && UP)
        asm("{\n\t.reg .b64 v, q, m;\n\t.reg .f32 one, up;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\t"
            "mov.f32 one, 0fBF800000;\n\tmov.f32 up, 0f43800000;\n\tmov.b64 m, {one, one};\n\tfma.rn.f32x2 v, q, m, v;\n\t"
            "mov.b64 m, {up, up};\n\tmul.rn.f32x2 v, v, m;\n\tmov.b64 {%0, %1}, v;\n\t}"
            : "+f"(lo), "+f"(hi) : "f"(__uint_as_float(p << 16)), "f"(__uint_as_float(p & 0xffff0000u)));
    else if (!last) {
        lo -= __uint_as_float(p << 16);
        hi -= __uint_as_float(p & 0xffff0000u);
    }
    return p;
}

__device__ __forceinline__ bool elect_one() {
    unsigned p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// first operand in tensor memory, second in shared memory; `down`: d = a b + d / 2^8
__device__ __forceinline__ void umma_from_tmem(unsigned d, unsigned a, unsigned long long b, unsigned idesc, unsigned accumulate, bool down) {
    if (down)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, 8;\n\t}"
                     ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// both operands in shared memory
__device__ __forceinline__ void umma_from_smem(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate, bool down) {
    if (down)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 8;\n\t}"
                     ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else umma_bf16(d, a, b, idesc, accumulate);
}
// (no memory clobber: loads of the next values may pass it; what follows waits with tcgen05.wait::st)
__device__ __forceinline__ void tmem_store8(unsigned addr, const unsigned (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]));
}
__device__ __forceinline__ void tmem_load8(unsigned addr, unsigned (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr));
}
// Sixteen values of a lane's row (their four quarters) into tensor memory: piece p at addr + p * step, eight columns each.
template <bool UP>
__device__ __forceinline__ void split16_to_tmem(float4 (&x)[4], unsigned addr, unsigned step) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
        unsigned v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = take_piece<UP>(x[i].x, x[i].y, p == PIECES - 1);
            v[2 * i + 1] = take_piece<UP>(x[i].z, x[i].w, p == PIECES - 1);
        }
        tmem_store8(addr + (unsigned)p * step, v);
    }
}
// Eight values into shared memory: piece p at dst + p * step, sixteen bytes each.
template <bool UP>
__device__ __forceinline__ void split8_to_smem(float4 a, float4 b, unsigned char* dst, int step) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
        const bool last = p == PIECES - 1;
        uint4 v;
        v.x = take_piece<UP>(a.x, a.y, last);
        v.y = take_piece<UP>(a.z, a.w, last);
        v.z = take_piece<UP>(b.x, b.y, last);
        v.w = take_piece<UP>(b.z, b.w, last);
        *reinterpret_cast<uint4*>(dst + p * step) = v;
    }
}
