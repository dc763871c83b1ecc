// MUL_MAT of packed quantized weights with 1..8 activation columns: the weights' integers, exact in f16, times the activations as
// two f16 numbers, with mma.sync straight from registers.
//
//   y[N, M] = W[K, N] . x[K, M]      values of src/core/ref/quant.cpp:30-108 and src/core/ref/ops.cpp:891-984
//
// A warp owns 256 weights of K (a unit) for the whole launch: its activations are B fragments in registers.  It walks down row
// tiles of 16 rows, whose bytes it copies to a ring of its own in shared memory (cp.async: whole lines of the row-major planes, no registers
// for what is in flight) and reads back as A fragments (ldmatrix: a matrix row is 16 bytes of a weight row).  The integers need no conversion:
// a bit field under the exponent of 1024 is an f16 number, and one packed addition takes 1024 and the format's offset (8, 32, 128) off, exactly; the unsigned
// ones of Q4_K (and OFFSET) stand under a zero exponent, subnormal numbers.  A block (32 weights, Q6_K 16) is multiplied into a fresh accumulator, which times the block's
// scale goes to f32 sums: no weight is scaled or rounded, and the tensor core's truncation sees 32 products at most.
//
// Activations: per column and unit one power of two brings the largest to [2^13, 2^14), then x = xh + 2^-11 xl, both f16: 22 bits, and because the low part is
// scaled up they are there down to 2^-35 of the largest (2^-31 for half of Q4_0's).  Not with M > 4 of Q4_K, 2^-24 there: it replaces kernels of 16-bit
// integers to the largest of 64 and would lose 0.4 us of 7.1 (4096 x 4096, 8 columns).  FINE: a third part likewise, which makes it the 24 bits of
// an f32 number down to 2^-37 of the largest, for the single columns of Q6_K that f32 kernels would serve otherwise (7168 x 8192: 15.9 us with two parts, 16.8 with three).
//   FINE    xh, xl and the third part of one token in three columns
//   M <= 4: the eight columns of an MMA are xh and xl of four tokens; M <= 8: two MMAs, xh and xl of eight
// Error against float64: 8e-8 to 1.3e-7, Q4_K 6e-7 to 1.4e-6, OFFSET 3e-7 (the integer column kernels 2e-5 to 6e-5, the split GEMM 5e-6, the f32 matvec of the vocabulary head 1e-6).
//
// The partial tiles of a CTA's units meet in shared memory and are added in the order of K; where K is longer than a CTA's 16 units, or more
// SMs have work that way, a cluster of two to six shares it and its CTAs read each other's sums.  No memory of the call, one launch.
//
// What bounds it: Q6_K the instructions that assemble 6 bits (the ALU pipe over 70 % busy in the loop), then 3 to 4 us of start (launch, activations from
// L2, their conversion) that one CTA per SM does not hide; K = 4096, N = 12288, 4 columns 13.3 us (with the offsets taken off afterwards 13.8, of that
// without the products 9.3, without the weights 11.8).
#include "sm100_common.cuh"
#include "sm100_layout.h"

namespace sm100 {

namespace {

constexpr int CO_WARPS = 16;    // at most
constexpr int CO_UNIT = 256;    // weights of K that a warp owns
constexpr int CO_MOST_K = 4 * CO_WARPS * CO_UNIT;

struct ColsArgs {
    const uint8_t * w;
    int64_t off1, off2, off3;   // planes behind the first
    const float * x;
    int64_t ldx;
    float * y;
    int64_t ldy;
    int m;
    int units;      // K / 256
    int tiles;      // 16-row tiles
    int wk, wr_log; // warps of a CTA: wk units x 2^wr_log row tiles
    int iters;      // row tiles of a warp
    int window;     // of them, as many whose partial sums meet at once
    uint32_t k1024; // CO_1024
};

__device__ __forceinline__ uint32_t co_smem(const void * p) { return (uint32_t) __cvta_generic_to_shared(p); }
__device__ __forceinline__ void co_cp16(uint32_t dst, const void * src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void co_cp4(uint32_t dst, const void * src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ uint32_t co_lds(uint32_t a) { uint32_t v; asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory"); return v; }
__device__ __forceinline__ uint4 co_lds4(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 co_lds4f(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void co_sts4f(uint32_t a, float x, float y, float z, float w) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
// four / two matrices of 8 rows x 16 bytes: lane 4 g + t receives word t of row g; lane 8 i + r gives the address of row r of matrix i
__device__ __forceinline__ void co_ldsm4(uint32_t (&v)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void co_ldsm2(uint32_t (&v)[2], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(a) : "memory");
}
// d = a b + c; d = a b
__device__ __forceinline__ void co_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void co_mma0(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t co_add2(uint32_t a, uint32_t b) { uint32_t d; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t h2(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ float co_half(uint32_t h) { return __half2float(__ushort_as_half((unsigned short) h)); }

// An integer below 1024 in the low bits of a half, under the exponent of 1024, is 1024 + the integer: no conversion.  Bits 4 .. 7 hold 16 times
// a nibble, whose step's activations are a 16th instead.  What the integers are too large by is subtracted from them, with the 1024, and not from the products: a
// weight of zero then multiplies by zero.  With the offset taken off afterwards, as the sum of x over the block times the scale, an activation 1e3
// times the others left an error of 6e-4 (Q4_0) in rows where its weight is zero, one of 1e5 times 9e-2.  The instruction that masks the bits also
// sets the exponent, and the sums need not be made: 4096 x 12288, us before / now: Q4_0 4 columns 10.1 / 10.3, 8 columns 13.5 / 13.1; Q8_0 8 columns 14.3 / 13.4;
// Q6_K 1 column 13.3 / 12.4, 4 columns 13.9 / 12.9, 8 columns 17.6 / 17.1.
// Q4_K, whose minima are part of the weights' values, has unsigned integers as subnormal numbers (they count 2^-24) and one more step over a
// unit: the sums of x over the blocks times the minima, small integers themselves.  Subnormal numbers in place of the signed ones' 1024: the tensor core's truncation
// costs more, 2e-7 instead of 1.2e-7 for a column of Q6_K and 4.4e-6 for eight of Q4_0 with an outlier of 3e6.
constexpr float CO_2_24 = 16777216.0f;
constexpr uint32_t CO_1024 = 0x64006400u;   // an argument of the launch: with two constants in it, masking and setting would be two instructions
// (a & MASK) | c in one instruction
template <uint32_t MASK>
__device__ __forceinline__ uint32_t co_pick(uint32_t a, uint32_t c) { uint32_t d; asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "n"(MASK), "r"(c)); return d; }
__device__ __forceinline__ uint32_t co_less1032(uint32_t a) { return co_add2(a, 0xe408e408u); }
__device__ __forceinline__ uint32_t co_less1152(uint32_t a) { return co_add2(a, 0xe480e480u); }

// B: the activations, per step of 16 weights pairs (0, 2) and (1, 3) of the lane's four, and where a format has them the sums over the blocks (2 t and 2 t + 1 of eight;
// 4 t and 4 t + 2, 4 t + 1 and 4 t + 3 of sixteen)
template <bool P4> struct CoB { uint32_t h[16][2], l[P4 ? 1 : 16][P4 ? 1 : 2]; uint32_t sum_h[2], sum_l, k1024; };

// What the low parts are multiplied by: as they are, the low part of an activation 2^-14 of the largest would be a subnormal number, with fewer bits (an activation
// 1e7 times the others left 2e-4 of them).  4096 x 12288, us before / now: Q8_0 4 columns 12.1 / 12.3, 8 columns 13.4 / 14.1; Q6_K 4 columns 12.9 / 13.4, 8 columns 17.1 / 17.7.
constexpr float CO_LOW = 2048.0f;

// acc = the products of a step; of two.  M <= 8: the low parts' come first, since the accumulator then is divided by what they are multiplied by (four
// multiplications; two accumulators would not leave enough registers).  M <= 4: the low parts have columns of their own.
template <bool P4>
__device__ __forceinline__ void co_block(float (&acc)[4], const uint32_t (&a)[4], const CoB<P4> & b, int s) {
    if constexpr (P4) {
        co_mma0(acc, a, b.h[s][0], b.h[s][1]);
    } else {
        co_mma0(acc, a, b.l[s][0], b.l[s][1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] *= 1.0f / CO_LOW;
        co_mma(acc, a, b.h[s][0], b.h[s][1]);
    }
}
template <bool P4>
__device__ __forceinline__ void co_block2(float (&acc)[4], const uint32_t (&a)[4], const uint32_t (&c)[4], const CoB<P4> & b, int s) {
    if constexpr (P4) {
        co_mma0(acc, a, b.h[s][0], b.h[s][1]);
    } else {
        co_mma0(acc, a, b.l[s][0], b.l[s][1]);
        co_mma(acc, c, b.l[s + 1][0], b.l[s + 1][1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] *= 1.0f / CO_LOW;
        co_mma(acc, a, b.h[s][0], b.h[s][1]);
    }
    co_mma(acc, c, b.h[s + 1][0], b.h[s + 1][1]);
}
// Q4_K, whose low parts are as they are with eight columns
template <bool P4>
__device__ __forceinline__ void co_mul0(float (&acc)[4], const uint32_t (&a)[4], const CoB<P4> & b, int s) {
    co_mma0(acc, a, b.h[s][0], b.h[s][1]);
    if constexpr (!P4) co_mma(acc, a, b.l[s][0], b.l[s][1]);
}
template <bool P4>
__device__ __forceinline__ void co_mul(float (&acc)[4], const uint32_t (&a)[4], const CoB<P4> & b, int s) {
    co_mma(acc, a, b.h[s][0], b.h[s][1]);
    if constexpr (!P4) co_mma(acc, a, b.l[s][0], b.l[s][1]);
}
__device__ __forceinline__ void co_scale(float (&sum)[4], const float (&acc)[4], float d0, float d1) {
    sum[0] = fmaf(d0, acc[0], sum[0]);
    sum[1] = fmaf(d0, acc[1], sum[1]);
    sum[2] = fmaf(d1, acc[2], sum[2]);
    sum[3] = fmaf(d1, acc[3], sum[3]);
}

// What a format does: a Cursor holds a lane's addresses of a unit in the row tile that is fetched next, fetch() copies that to a slot (cp.async) and goes
// `step` tiles on, run() multiplies.  sum = 1 / COUNT times the products.
// Q4_0 and Q8_0: per row the unit's quants and its eight f16 scales
template <bool Q8>
struct CoB32 {
    static constexpr bool FINE = false, OFFSET = false;
    static constexpr int QB = Q8 ? 256 : 128, PITCH = QB + 16, SLOT = 16 * PITCH, SLOTS = Q8 ? 2 : 4, TABLE = 0;
    static constexpr int BLOCKS = 0;
    static constexpr bool SCALED = true;
    static constexpr float COUNT = 1.0f;
    struct Cursor { const uint8_t * q; const uint8_t * d; };
    __device__ static __forceinline__ int k_of(int s) { return 16 * s; }
    __device__ static __forceinline__ bool sixteenth(int s) { return !Q8 && (s & 1); }
    static constexpr int PIECES = QB / 16, ROWS = 32 / PIECES;   // a warp's copy of 16 bytes a lane: ROWS rows
    __device__ static __forceinline__ void init(Cursor & c, const ColsArgs & g, int rt, int unit, int lane) {
        c.q = g.w + (((int64_t) rt * 16 + lane / PIECES) * g.units + unit) * QB + (lane % PIECES) * 16;
        c.d = g.w + g.off1 + (((int64_t) rt * 16 + (lane & 15)) * g.units + unit) * 16;
    }
    __device__ static __forceinline__ void fetch(Cursor & c, const ColsArgs & g, uint32_t slot, int64_t step, int lane) {
        const uint32_t to = slot + (lane / PIECES) * PITCH + (lane % PIECES) * 16;
        const uint8_t * q = c.q;
#pragma unroll
        for (int i = 0; i < 16 / ROWS; ++i) {
            co_cp16(to + i * ROWS * PITCH, q);
            q += (int64_t) g.units * (ROWS * QB);
        }
        if (lane < 16) co_cp16(slot + lane * PITCH + QB, c.d);
        c.q += step * QB;
        c.d += step * 16;
    }
    template <bool P4>
    __device__ static __forceinline__ void run(uint32_t slot, uint32_t, int, int lane, const CoB<P4> & b, float (&sum)[4]) {
        // matrices: rows 0-7, rows 8-15 of one 16-byte piece, then of the next
        const uint32_t at = slot + (lane & 15) * PITCH + (lane >> 4) * 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j] = 0.f;
        const uint4 s0 = co_lds4(slot + (lane >> 2) * PITCH + QB), s1 = co_lds4(slot + (8 + (lane >> 2)) * PITCH + QB);
        const uint32_t d0[4] = {s0.x, s0.y, s0.z, s0.w}, d1[4] = {s1.x, s1.y, s1.z, s1.w};
        auto scale = [&](const float (&acc)[4], int blk) {
            co_scale(sum, acc, co_half(blk & 1 ? d0[blk >> 1] >> 16 : d0[blk >> 1] & 0xffffu), co_half(blk & 1 ? d1[blk >> 1] >> 16 : d1[blk >> 1] & 0xffffu));
        };
#pragma unroll
        for (int i = 0; i < QB / 32; ++i) {
            uint32_t v[4];
            co_ldsm4(v, at + 32 * i);
            const uint32_t u[4] = {v[0] >> 8, v[1] >> 8, v[2] >> 8, v[3] >> 8};
            float acc[4];
            if constexpr (Q8) {   // a block: its two pieces; the signed bytes, 1024 + 128 added and taken off again
                const uint32_t k1152 = b.k1024 ^ 0x00800080u;
                auto sb = [&](uint32_t q) { return co_less1152((q & 0x00ff00ffu) ^ k1152); };
                const uint32_t a[4] = {sb(v[0]), sb(v[1]), sb(u[0]), sb(u[1])}, c[4] = {sb(v[2]), sb(v[3]), sb(u[2]), sb(u[3])};
                co_block2<P4>(acc, a, c, b, 2 * i);
                scale(acc, i);
            } else {              // two blocks of 16 bytes
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    auto lo = [&](uint32_t q) { return co_less1032(co_pick<0x000f000fu>(q, b.k1024)); };
                    auto hi = [&](uint32_t q) { return co_less1152(co_pick<0x00f000f0u>(q, b.k1024)); };
                    const uint32_t a[4] = {lo(v[2 * e]), lo(v[2 * e + 1]), lo(u[2 * e]), lo(u[2 * e + 1])};
                    const uint32_t c[4] = {hi(v[2 * e]), hi(v[2 * e + 1]), hi(u[2 * e]), hi(u[2 * e + 1])};
                    co_block2<P4>(acc, a, c, b, 4 * i + 2 * e);
                    scale(acc, 2 * i + e);
                }
            }
        }
    }
};

// Q4_K: four lane-ordered tiles of 512 bytes, then the rows' headers.  Table: d sc of [16 rows][8 sub-blocks], padded to 12; of the odd ones,
// whose nibbles count 16, a 16th.
struct CoQ4K {
    static constexpr bool FINE = false, OFFSET = false;
    static constexpr int SLOT = 4 * 512 + 256, SLOTS = 4, TABLE = 16 * 12 * 4;
    static constexpr int BLOCKS = 8;   // of a unit whose sums of x are wanted
    static constexpr bool SCALED = false;
    static constexpr float COUNT = CO_2_24;
    struct Cursor { const uint8_t * q; const uint8_t * h; };
    __device__ static __forceinline__ int k_of(int s) { return 16 * s; }
    __device__ static __forceinline__ bool sixteenth(int) { return false; }
    __device__ static __forceinline__ void init(Cursor & c, const ColsArgs & g, int rt, int unit, int lane) {
        c.q = g.w + ((int64_t) rt * g.units + unit) * 2048 + lane * 16;
        c.h = g.w + g.off1 + (((int64_t) rt * 16 + (lane & 15)) * g.units + unit) * 16;
    }
    __device__ static __forceinline__ void fetch(Cursor & c, const ColsArgs & g, uint32_t slot, int64_t step, int lane) {
#pragma unroll
        for (int i = 0; i < 4; ++i) co_cp16(slot + i * 512 + lane * 16, c.q + i * 512);
        if (lane < 16) co_cp16(slot + 2048 + lane * 16, c.h);
        c.q += step * 128;
        c.h += step * 16;
    }
    // the 24-bit field p of a header: sc | m << 6 of sub-block 2 p, the same of 2 p + 1 from bit 12
    __device__ static __forceinline__ uint32_t field(uint32_t head, int p) {   // head: address of the header
        const uint32_t lo = co_lds(head + 4 + (p * 3 & ~3)), hi = co_lds(head + 4 + ((p * 3 + 2) & ~3));
        return __funnelshift_r(lo, hi, (p * 3 & 3) * 8);
    }
    template <bool P4>
    __device__ static __forceinline__ void run(uint32_t slot, uint32_t table, int, int lane, const CoB<P4> & b, float (&sum)[4]) {
        const int gr = lane >> 2, t = lane & 3;
        {   // lane (g, t): scales and minima of sub-blocks 2 t and 2 t + 1 of rows g and g + 8; the minima times the sums of x
            const uint32_t h0 = slot + 2048 + gr * 16, h1 = h0 + 128, f0 = field(h0, t), f1 = field(h1, t), w0 = co_lds(h0), w1 = co_lds(h1);
            const float d0 = co_half(w0 & 0xffffu), d1 = co_half(w1 & 0xffffu), m0 = -32.0f * co_half(w0 >> 16), m1 = -32.0f * co_half(w1 >> 16);
            const uint32_t to = table + gr * 48 + t * 8;
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(d0 * (float) (f0 & 63u)), "f"(d0 * 0.0625f * (float) ((f0 >> 12) & 63u)) : "memory");
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(to + 8 * 48), "f"(d1 * (float) (f1 & 63u)), "f"(d1 * 0.0625f * (float) ((f1 >> 12) & 63u)) : "memory");
            const uint32_t a[4] = {((f0 >> 6) & 63u) | ((f0 >> 2) & 0x003f0000u), ((f1 >> 6) & 63u) | ((f1 >> 2) & 0x003f0000u), 0u, 0u};
            float acc[4];
            co_mma0(acc, a, b.sum_h[0], 0u);
            if constexpr (!P4) co_mma(acc, a, b.sum_l, 0u);
            sum[0] = m0 * acc[0]; sum[1] = m0 * acc[1]; sum[2] = m1 * acc[2]; sum[3] = m1 * acc[3];
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint4 q = co_lds4(slot + c * 512 + lane * 16);
            float2 e0, e1;
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(e0.x), "=f"(e0.y) : "r"(table + gr * 48 + c * 8) : "memory");
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(e1.x), "=f"(e1.y) : "r"(table + (gr + 8) * 48 + c * 8) : "memory");
            const uint32_t v[2][2] = {{q.x, q.z}, {q.y, q.w}};   // [half of the sub-block][row]
            float lo[4], hi[4];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const uint32_t v0 = v[e][0], v1 = v[e][1], u0 = v0 >> 8, u1 = v1 >> 8;
                const uint32_t a[4] = {v0 & 0x000f000fu, v1 & 0x000f000fu, u0 & 0x000f000fu, u1 & 0x000f000fu};
                const uint32_t d[4] = {v0 & 0x00f000f0u, v1 & 0x00f000f0u, u0 & 0x00f000f0u, u1 & 0x00f000f0u};
                if (e == 0) {
                    co_mul0<P4>(lo, a, b, 4 * c);
                    co_mul0<P4>(hi, d, b, 4 * c + 2);
                } else {
                    co_mul<P4>(lo, a, b, 4 * c + 1);
                    co_mul<P4>(hi, d, b, 4 * c + 3);
                }
            }
            co_scale(sum, lo, e0.x, e1.x);
            co_scale(sum, hi, e0.y, e1.y);
        }
    }
};

// Q6_K: per row 128 bytes of nibbles, 64 of bit pairs, 16 scales; then the words that hold the rows' d.  Table: d sc of
// [16 rows][16 groups], padded to 20; of every third and fourth group, whose integers count 16, a 16th.
// OFFSET: the integers stay unsigned subnormal numbers, 32 times the sums of x comes off afterwards, and low parts are as they are: for the single columns that 16-bit integers
// served before.  It is the more accurate of these two beside large activations (rows whose weights there are zero, at 1e3 / 1e5 times the others: 1e-4 / 0.02, the integers
// 2e-3 / 0.2), and its bits stay, since a decode step makes 6e-5 of its logits of any other rounding here: every layer behind it rounds to 16 bits.
enum { Q6K_TWO_PARTS, Q6K_FINE, Q6K_OFFSET };
template <int FORM>
struct CoQ6K {
    static constexpr bool FINE = FORM == Q6K_FINE, OFFSET = FORM == Q6K_OFFSET;
    static constexpr int PITCH = 208, SLOT = 16 * PITCH + 64, SLOTS = 3, TABLE = 16 * 20 * 4;
    static constexpr int BLOCKS = OFFSET ? 16 : 0;
    static constexpr bool SCALED = !OFFSET;
    static constexpr float COUNT = OFFSET ? CO_2_24 : 1.0f;
    struct Cursor { const uint8_t * q; const uint8_t * x; const uint8_t * s; const uint8_t * d; };
    __device__ static __forceinline__ int k_of(int s) { return 128 * (s >> 3) + 16 * ((s >> 2) & 1) + 32 * (s & 3); }
    __device__ static __forceinline__ bool sixteenth(int) { return false; }
    __device__ static __forceinline__ void init(Cursor & c, const ColsArgs & g, int rt, int unit, int lane) {
        const int64_t row0 = (int64_t) rt * 16, blk = (row0 + (lane & 15)) * g.units + unit;
        c.q = g.w + ((row0 + (lane >> 3)) * g.units + unit) * 128 + (lane & 7) * 16;
        c.x = g.w + g.off1 + ((row0 + (lane >> 2)) * g.units + unit) * 64 + (lane & 3) * 16;
        c.s = g.w + g.off2 + blk * 16;
        c.d = g.w + g.off3 + (blk & ~(int64_t) 1) * 2;   // a word; both its blocks lie inside the plane (whole tiles have an even number of blocks)
    }
    __device__ static __forceinline__ void fetch(Cursor & c, const ColsArgs & g, uint32_t slot, int64_t step, int lane) {
        const uint32_t tq = slot + (lane >> 3) * PITCH + (lane & 7) * 16, tx = slot + (lane >> 2) * PITCH + 128 + (lane & 3) * 16;
        const uint8_t * q = c.q;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            co_cp16(tq + i * 4 * PITCH, q);
            q += (int64_t) g.units * 512;
        }
        co_cp16(tx, c.x);
        co_cp16(tx + 8 * PITCH, c.x + (int64_t) g.units * 512);
        if (lane < 16) {
            co_cp16(slot + lane * PITCH + 192, c.s);
            co_cp4(slot + 16 * PITCH + lane * 4, c.d);
        }
        c.q += step * 128;
        c.x += step * 64;
        c.s += step * 16;
        c.d += step * 2;
    }
    template <bool P4>
    __device__ static __forceinline__ void run(uint32_t slot, uint32_t table, int odd, int lane, const CoB<P4> & b, float (&sum)[4]) {
        const int gr = lane >> 2, t = lane & 3;
        const uint32_t at = slot + (lane & 15) * PITCH;   // matrices of rows 0-7 and 8-15
        {   // lane (g, t): scales 4 t .. 4 t + 3 of rows g and g + 8, for the table and (OFFSET), as f16 integers, times the sums of x
            uint32_t v[2];
            co_ldsm2(v, at + 192);
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            if constexpr (OFFSET) {
                const uint32_t a[4] = {co_less1152((v[0] & 0x00ff00ffu) ^ 0x64806480u), co_less1152((v[1] & 0x00ff00ffu) ^ 0x64806480u),
                                       co_less1152(((v[0] >> 8) & 0x00ff00ffu) ^ 0x64806480u), co_less1152(((v[1] >> 8) & 0x00ff00ffu) ^ 0x64806480u)};
                co_mma0(acc, a, b.sum_h[0], b.sum_h[1]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float d = co_half(co_lds(slot + 16 * PITCH + (gr + 8 * h) * 4) >> ((odd >> gr & 1) * 16) & 0xffffu);   // `odd`: bit r = row r's block has an odd number (row r + 8 like row r)
                const int w = (int) v[h];
                const float d16 = OFFSET ? d : d * 0.0625f;
                co_sts4f(table + (gr + 8 * h) * 80 + t * 16, d * (float) (w << 24 >> 24), d * (float) (w << 16 >> 24), d16 * (float) (w << 8 >> 24), d16 * (float) (w >> 24));
                sum[2 * h] = OFFSET ? d * (-1024.0f / CO_2_24) * acc[2 * h] : 0.f;
                sum[2 * h + 1] = OFFSET ? d * (-1024.0f / CO_2_24) * acc[2 * h + 1] : 0.f;
            }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c) {   // the block's four units of the packed layout
            const float4 e0 = co_lds4f(table + gr * 80 + c * 16), e1 = co_lds4f(table + (gr + 8) * 80 + c * 16);
            uint32_t a[4][4];   // [group][fragment word]
            uint32_t n[4], x[2];
            const uint32_t k1024 = OFFSET ? 0u : b.k1024;
            co_ldsm4(n, at + 32 * c + (lane >> 4) * 16);
            co_ldsm2(x, at + 128 + 16 * c);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t n0 = n[h], n1 = n[2 + h], m0 = n0 >> 8, m1 = n1 >> 8, y = x[h] >> 8, xa = x[h] << 4, xb = x[h] << 2, ya = y << 4, yb = y << 2;
                a[0][h] = co_pick<0x000f000fu>(n0, co_pick<0x00300030u>(xa, k1024));
                a[0][2 + h] = co_pick<0x000f000fu>(m0, co_pick<0x00300030u>(ya, k1024));
                a[1][h] = co_pick<0x000f000fu>(n1, co_pick<0x00300030u>(xb, k1024));
                a[1][2 + h] = co_pick<0x000f000fu>(m1, co_pick<0x00300030u>(yb, k1024));
                a[2][h] = co_pick<0x00f000f0u>(n0, co_pick<0x03000300u>(xa, k1024));
                a[2][2 + h] = co_pick<0x00f000f0u>(m0, co_pick<0x03000300u>(ya, k1024));
                a[3][h] = co_pick<0x00f000f0u>(n1, co_pick<0x03000300u>(xb, k1024));
                a[3][2 + h] = co_pick<0x00f000f0u>(m1, co_pick<0x03000300u>(yb, k1024));
            }
            if constexpr (!OFFSET) {   // 1024 + q - 1056, 1024 + 16 q - 1536
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[j][i] = co_add2(a[j][i], j < 2 ? 0xe420e420u : 0xe600e600u);
            }
            const float s0[4] = {e0.x, e0.y, e0.z, e0.w}, s1[4] = {e1.x, e1.y, e1.z, e1.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float acc[4];
                co_block<P4>(acc, a[j], b, 4 * c + j);
                co_scale(sum, acc, s0[j], s1[j]);
            }
        }
    }
};

template <typename F, bool P4>
__global__ void __launch_bounds__(32 * CO_WARPS, 1) quant_cols(const ColsArgs g) {
    constexpr int COLS = P4 ? 4 : 8, TILE = COLS * 16;   // floats of a partial tile: [column][row]
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3;
    const int kp = warp % g.wk, rg = warp / g.wk, wr = 1 << g.wr_log;
    uint32_t rank, csize;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
    const int clusters = (int) (gridDim.x / csize), cid = (int) (blockIdx.x / csize);
    const int unit0 = (int) (rank * g.units / csize), my_units = (int) ((rank + 1) * g.units / csize) - unit0, unit = unit0 + kp;
    const bool live = kp < my_units;
    const uint32_t ring = co_smem(smem_raw) + warp * (F::SLOTS * F::SLOT + F::TABLE), table = ring + F::SLOTS * F::SLOT;
    const uint32_t red0 = co_smem(smem_raw) + (blockDim.x >> 5) * (F::SLOTS * F::SLOT + F::TABLE);
    const uint32_t red_bytes = (uint32_t) (g.wk * TILE * 4 * g.window) << g.wr_log;   // per parity: [tile of the window][row group][unit][TILE]
    const bool twice = g.window < g.iters;   // two sets of partial sums, in turn
    const uint32_t fold0 = red0 + (twice ? 2 : 1) * red_bytes, fold_bytes = (uint32_t) (g.window * TILE * 4) << g.wr_log;

    // the warp's tiles: (cid + clusters i) wr + rg
    const int tile0 = (cid << g.wr_log) + rg, tile_step = clusters << g.wr_log;
    const int my_tiles = live && tile0 < g.tiles ? (g.tiles - tile0 + tile_step - 1) / tile_step : 0;
    const int64_t step = (int64_t) tile_step * 16 * g.units;   // in blocks of 256 weights
    typename F::Cursor cur;
    F::init(cur, g, tile0 < g.tiles ? tile0 : 0, live ? unit : 0, lane);
    auto fetch = [&](int i, int slot) {
        if (i < my_tiles) F::fetch(cur, g, ring + slot * F::SLOT, step, lane);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < F::SLOTS - 1; ++i) fetch(i, i);

    pdl_wait();
    // ---- activations: lane (g, t) holds column g's weights k_of(s) + 4 t .. + 3 of each step (M <= 4: column g % 4, high parts for g < 4, low parts beyond) ----
    CoB<P4> b;
    b.k1024 = g.k1024;
    float back[2];   // of the lane's two result columns: 1 / scale
    {
        const int col = P4 ? (lane >> 2) & 3 : lane >> 2;
        const bool lo_lane = P4 && lane >= 16;
        const float * src = g.x + (int64_t) (col < g.m ? col : 0) * g.ldx + (int64_t) (live ? unit : 0) * CO_UNIT + 4 * t;
        float4 v[16];
#pragma unroll
        for (int s = 0; s < 16; ++s) v[s] = __ldcg(reinterpret_cast<const float4 *>(src + F::k_of(s)));
        float top = 0.f;   // a NaN does not show here and is still there below
#pragma unroll
        for (int s = 0; s < 16; ++s) top = fmaxf(fmaxf(fmaxf(top, fabsf(v[s].x)), fmaxf(fabsf(v[s].y), fabsf(v[s].z))), fabsf(v[s].w));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        bool infinite = false;
        if constexpr (F::FINE) {   // as f32 gives it: an infinity times its weight.  It is left out of the scale and of the lower parts; every lane has the same column
            infinite = top == INFINITY;
            if (infinite) {
                auto finite = [](float & f) { f = fabsf(f) == INFINITY ? 0.f : f; return fabsf(f); };
                top = 0.f;
#pragma unroll
                for (int s = 0; s < 16; ++s) top = fmaxf(fmaxf(fmaxf(top, finite(v[s].x)), fmaxf(finite(v[s].y), finite(v[s].z))), finite(v[s].w));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            }
        }
        // the largest to [2^13, 2^14), subnormal numbers as far as 2^126 brings them; infinities as they are
        const int e = __float_as_int(top) >> 23;
        int sh = e == 255 ? 0 : 13 + 127 - e;
        sh = sh > 126 ? 126 : sh;   // >= 13 - 127
        // FINE: the columns that nobody reads are zero, the fewer bits toggle
        const float scale = F::FINE && ((lane >> 2) & 3) > (lo_lane ? 0 : 1) ? 0.f : __int_as_float((127 + sh) << 23), inv = __int_as_float((127 - sh) << 23);
        back[0] = __shfl_sync(0xffffffffu, inv, P4 ? (8 * t) & 15 : 8 * t);
        back[1] = __shfl_sync(0xffffffffu, inv, P4 ? (8 * t + 4) & 15 : 8 * t + 4);
        constexpr bool SCALED = (P4 && !F::OFFSET) || F::SCALED;
        constexpr float LOW = SCALED ? CO_LOW : 1.0f;
        // f, or what it is less its high part, scaled.  Two numbers an instruction (Q4_0 4096 x 12288, 4 columns: 10.5 us with one, 10.3)
        // FINE: lanes 0..3 hold the first part, 16..19 the second, 4..7 the third, which takes another step.
        const bool third = F::FINE && (lane >> 2) == 1, low = lo_lane || third || !P4;
        const float2 up3 = third ? make_float2(CO_LOW, CO_LOW) : make_float2(1.f, 1.f), less3 = third ? make_float2(-CO_LOW, -CO_LOW) : make_float2(0.f, 0.f);
        const float2 up = low ? make_float2(LOW, LOW) : make_float2(1.f, 1.f), less = low ? make_float2(-LOW, -LOW) : make_float2(0.f, 0.f);
        const __half2 z = __float2half2_rn(0.0625f);
        float sums[F::BLOCKS ? F::BLOCKS : 1];
#pragma unroll
        for (int s = 0; s < 16; ++s) {
            const float sc = F::sixteenth(s) ? scale * 0.0625f : scale;
            const float2 f0 = __fmul2_rn(make_float2(v[s].x, v[s].y), make_float2(sc, sc)), f1 = __fmul2_rn(make_float2(v[s].z, v[s].w), make_float2(sc, sc));
            if constexpr (F::BLOCKS > 0) {
                constexpr int PER = 16 / (F::BLOCKS ? F::BLOCKS : 16);
                const float q = (f0.x + f1.x) + (f0.y + f1.y);
                sums[s / PER] = s % PER ? sums[s / PER] + q : q;
            }
            const __half2 hx = __floats2half2_rn(f0.x, f1.x), hy = __floats2half2_rn(f0.y, f1.y);   // pairs (0, 2) and (1, 3)
            const float2 rx = __half22float2(hx), ry = __half22float2(hy);
            float2 u0, u1;
            if constexpr (SCALED || P4) {
                u0 = __ffma2_rn(make_float2(rx.x, ry.x), less, __fmul2_rn(f0, up));
                u1 = __ffma2_rn(make_float2(rx.y, ry.y), less, __fmul2_rn(f1, up));
            } else {
                u0 = __ffma2_rn(make_float2(rx.x, ry.x), make_float2(-1.f, -1.f), f0);
                u1 = __ffma2_rn(make_float2(rx.y, ry.y), make_float2(-1.f, -1.f), f1);
            }
            if constexpr (F::FINE) {
                const float2 qx = __half22float2(__floats2half2_rn(u0.x, u1.x)), qy = __half22float2(__floats2half2_rn(u0.y, u1.y));
                u0 = __ffma2_rn(make_float2(qx.x, qy.x), less3, __fmul2_rn(u0, up3));
                u1 = __ffma2_rn(make_float2(qx.y, qy.y), less3, __fmul2_rn(u1, up3));
            }
            uint32_t ux = h2(__floats2half2_rn(u0.x, u1.x)), uy = h2(__floats2half2_rn(u0.y, u1.y));
            if (F::OFFSET && (s & 2)) {
                ux = h2(__hmul2(*reinterpret_cast<__half2 *>(&ux), z));
                uy = h2(__hmul2(*reinterpret_cast<__half2 *>(&uy), z));
            }
            if constexpr (P4) {
                b.h[s][0] = ux;
                b.h[s][1] = uy;
            } else {
                b.h[s][0] = h2(hx);
                b.h[s][1] = h2(hy);
                b.l[s][0] = ux;
                b.l[s][1] = uy;
            }
        }
        if constexpr (F::FINE) {
            if (infinite && lane < 4) {
                auto put = [](uint32_t & h, float a, float c) {
                    if (fabsf(a) == INFINITY) h = (h & 0xffff0000u) | (a > 0.f ? 0x7c00u : 0xfc00u);
                    if (fabsf(c) == INFINITY) h = (h & 0x0000ffffu) | (c > 0.f ? 0x7c000000u : 0xfc000000u);
                };
#pragma unroll
                for (int s = 0; s < 16; ++s) {
                    const float4 f = __ldcg(reinterpret_cast<const float4 *>(src + F::k_of(s)));
                    put(b.h[s][0], f.x, f.z);
                    put(b.h[s][1], f.y, f.w);
                }
            }
        }
        if constexpr (F::BLOCKS > 0) {   // over the lanes that share a block, a 32nd of them
#pragma unroll
            for (int i = 0; i < F::BLOCKS; ++i) {
                sums[i] += __shfl_xor_sync(0xffffffffu, sums[i], 1);
                sums[i] += __shfl_xor_sync(0xffffffffu, sums[i], 2);
                sums[i] *= 0.03125f;
            }
#pragma unroll
            for (int i = 0; i < F::BLOCKS / 8; ++i) {
                float a[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    constexpr int N = F::BLOCKS / 4;   // blocks of a lane
                    const int o = F::BLOCKS == 8 ? j : 2 * j + i;
                    a[j] = t == 0 ? sums[o] : t == 1 ? sums[N + o] : t == 2 ? sums[2 * N + o] : sums[3 * N + o];
                }
                const __half2 hh = __floats2half2_rn(a[0], a[1]);
                const float2 r = __half22float2(hh);
                const __half2 ll = __floats2half2_rn((a[0] - r.x) * LOW, (a[1] - r.y) * LOW);
                b.sum_h[i] = h2(lo_lane ? ll : hh);
                if constexpr (!P4) b.sum_l = h2(ll);
            }
        }
    }
    pdl_launch_dependents();

    int slot = 0;
    // parity of the rows' block numbers, (16 rt + r) units + unit
    const int odd = g.units & 1 ? (unit & 1 ? 0x5555 : 0xaaaa) : (unit & 1 ? 0xffff : 0);
    int parity = 0;
    for (int i0 = 0; i0 < g.iters; i0 += g.window, parity ^= 1) {
#pragma unroll 1
        for (int i = i0; i < i0 + g.window; ++i) {
            // the slot that was read last (one iteration ago) is free: every lane is past it
            __syncwarp();
            fetch(i + F::SLOTS - 1, slot == 0 ? F::SLOTS - 1 : slot - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(F::SLOTS - 1) : "memory");
            __syncwarp();
            if (i < my_tiles) {
                float sum[4];
                F::template run<P4>(ring + slot * F::SLOT, table, odd, lane, b, sum);
                const uint32_t at = red0 + parity * red_bytes + 4u * (uint32_t) ((((i - i0) << g.wr_log) + rg) * g.wk + kp) * TILE;
                if constexpr (P4) {   // high and low parts' products: columns j and j + 4 (lanes t and t + 2)
#pragma unroll
                    for (int j = 0; j < 4; ++j) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], 2) * (F::OFFSET ? 1.0f : 1.0f / CO_LOW);
                }
                if constexpr (F::FINE) {   // the third part's products: column 1
                    sum[0] = fmaf(sum[1], 1.0f / (CO_LOW * CO_LOW), sum[0]);
                    sum[2] = fmaf(sum[3], 1.0f / (CO_LOW * CO_LOW), sum[2]);
                }
                if (!P4 || t < 2) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 4u * (uint32_t) ((2 * t + (j & 1)) * 16 + (lane >> 2) + 8 * (j >> 1))), "f"(sum[j] * F::COUNT * back[j & 1]) : "memory");
                }
            }
            slot = slot + 1 == F::SLOTS ? 0 : slot + 1;
        }
        __syncthreads();
        // ---- the window's tiles: units in the order of K, then the CTAs of the cluster ----
        const int outs = g.window * TILE << g.wr_log;
        auto store = [&](int e, float v) {
            const int tw = e / TILE, in = e % TILE, i = i0 + (tw >> g.wr_log), rt = ((cid + clusters * i) << g.wr_log) + (tw & (wr - 1));
            if (i < g.iters && rt < g.tiles) g.y[(int64_t) (in >> 4) * g.ldy + rt * 16 + (in & 15)] = v;
        };
        for (int e = threadIdx.x; e < outs; e += blockDim.x) {
            const int tw = e / TILE, in = e % TILE;
            if ((in >> 4) >= g.m) continue;
            const uint32_t at = red0 + parity * red_bytes + 4u * (uint32_t) (tw * g.wk * TILE + in);
            float v = 0.f;
#pragma unroll 8
            for (int p = 0; p < my_units; ++p) v += __uint_as_float(co_lds(at + 4u * (uint32_t) (p * TILE)));
            if (csize == 1) store(e, v);
            else asm volatile("st.shared.f32 [%0], %1;" ::"r"(fold0 + parity * fold_bytes + 4u * (uint32_t) e), "f"(v) : "memory");
        }
        if (csize > 1) {
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
            for (int e = (int) (rank * blockDim.x) + threadIdx.x; e < outs; e += (int) (csize * blockDim.x)) {
                if ((e % TILE >> 4) >= g.m) continue;
                const uint32_t at = fold0 + parity * fold_bytes + 4u * (uint32_t) e;
                float v = 0.f;
                for (uint32_t r = 0; r < csize; ++r) {
                    float u;
                    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}" : "=f"(u) : "r"(at), "r"(r) : "memory");
                    v += u;
                }
                store(e, v);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (csize > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // nobody leaves while another reads its sums
}

// How K and the rows are dealt: a cluster of `cluster` CTAs (one per SM) shares K, wk units each; a CTA takes 2^wr_log row tiles at a time.
struct ColsPlan { int cluster, wk, wr_log, at_once; };

// The time of a plan goes with the row tiles that a warp walks down (`iters`) and with the warps that share an SM while it does so (fewer than six are no faster each),
// plus start, which goes with the warps too, and the exchange of a cluster; a CTA more in the cluster counts 5 %.  Over 3623 products (K 256 .. 14336, N 1024 .. 32768, the four
// formats, 2, 4 and 8 columns) this choice is 1.3 % off the best plan on average, 133 of them by over 10 %.  A sum without start, and with little for a cluster, was 3.1 % off and
// 432, up to 1.64 times the integer kernel's time with Q4_K.  8 columns of that, us, by that sum's plan / this one's / in the integer kernel: 768 x 11264 9.5 / 5.8 / 5.8;
// 2048 x 2560 5.7 / 4.6 / 4.3; 4352 x 4096 10.3 / 8.4 / 7.3; 6144 x 4096 11.0 / 9.2 / 8.6.
// at_once: clusters that run at a time where every CTA has an SM of its own; SMs lie in groups that a cluster does not cross, so it is
// fewer than 148 / cluster (a 7 x 17 grid took twice as long as one of 15).
inline bool plan_cols(int units, int tiles, ColsPlan & p) {
    static const int most[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    int64_t best = INT64_MAX;
    for (int c = 1; c <= 8 && c <= units; ++c) {
        const int wk = (units + c - 1) / c, at_once = most[c] * sm_count() / 148;
        if (wk > CO_WARPS || at_once < 2) continue;
        for (int wl = 0; wk << wl <= CO_WARPS; ++wl) {
            const int64_t groups = (tiles + (1 << wl) - 1) >> wl, iters = (groups + at_once - 1) / at_once;
            const int warps = wk << wl;
            // a plan that needs every place for a cluster of three or more has to wait for one
            const int64_t counted = c > 2 ? (groups + at_once - 2) / (at_once - 1) : iters;
            const int64_t cost = counted * ((warps > 6 ? warps : 6) + 6) * (19 + c) + 40 * warps + (c > 1 ? 320 + 40 * c : 0);
            if (cost < best || (cost == best && p.cluster == c)) { best = cost; p = {c, wk, wl, at_once}; }
        }
    }
    return best != INT64_MAX;
}

template <typename F, bool P4>
int launch_cols(cudaStream_t s, ColsArgs g) {
    ColsPlan plan;
    if (!plan_cols(g.units, g.tiles, plan)) return fail(ST_BACKEND, "mul_mat: rows too long for the column kernel");
    const int wr = 1 << plan.wr_log, groups = (g.tiles + wr - 1) / wr, clusters = groups < plan.at_once ? groups : plan.at_once, warps = plan.wk * wr;
    g.wk = plan.wk;
    g.wr_log = plan.wr_log;
    g.iters = (groups + clusters - 1) / clusters;
    // partial sums of all row tiles at once where they fit (a meeting per two tiles instead of per six: 4096 x 12288, Q6_K, 4 columns
    // 14.8 us, 13.8; 12288 x 4096 18.0, 15.7), else two sets of even windows
    constexpr int MOST = 226 << 10;
    const int ring = warps * (F::SLOTS * F::SLOT + F::TABLE), tile = wr * (plan.wk + (plan.cluster > 1 ? 1 : 0)) * (P4 ? 64 : 128) * 4, room = MOST - ring;
    g.window = g.iters;
    if (g.iters > room / tile) {
        const int fit = room / (2 * tile), n = (g.iters + fit - 1) / fit;   // fit >= 1: 16 units and two sets of a tile's sums take 34 KB beside the largest ring
        g.window = (g.iters + n - 1) / n;
    }
    const int smem = ring + (g.window < g.iters ? 2 : 1) * g.window * tile;
    auto kernel = quant_cols<F, P4>;
    SM100_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST));
    return launch_cluster(kernel, dim3((unsigned) (clusters * plan.cluster)), dim3((unsigned) (32 * warps)), (size_t) smem, s, (unsigned) plan.cluster, g);
}

template <typename F>
int launch_cols(cudaStream_t s, const ColsArgs & g) { return g.m <= 4 ? launch_cols<F, true>(s, g) : launch_cols<F, false>(s, g); }

}  // namespace

// The full 16-row tiles of a packed tensor, 1..8 columns; `fine`: one column of Q6_K with the 24 bits of its activations, where f32 kernels would serve it.  *handled = false (and ST_OK) for
// rows that are not whole units, or longer than four CTAs' units: larger clusters leave too many SMs idle (28672 x 8192, Q6_K, 1 column: 122 us with
// clusters of 7, the f32 kernel 66).
int quant_cols_tiles(cudaStream_t s, int dtype, const void * w, int64_t k, int64_t n, const float * x, int64_t ldx, int64_t m, float * y, int64_t ldy, bool fine, bool * handled) {
    *handled = false;
    if (k % CO_UNIT != 0 || k > CO_MOST_K || n < 16 || n > INT32_MAX - 16 || m < 1 || m > 8) return ST_OK;
    if ((((uintptr_t) x) & 15) != 0 || (m > 1 && ldx % 4 != 0) || (((uintptr_t) w) & 31) != 0) return ST_OK;
    ColsArgs g = {};
    const Planes P = planes_for(dtype, n, k);
    g.w = (const uint8_t *) w;
    g.off1 = P.off[1];
    g.off2 = P.off[2];
    g.off3 = P.off[3];
    g.x = x;
    g.ldx = ldx;
    g.y = y;
    g.ldy = ldy;
    g.m = (int) m;
    g.units = (int) (k / CO_UNIT);
    g.tiles = (int) (n / 16);
    g.k1024 = CO_1024;
    *handled = true;
    switch (dtype) {
        case DT_Q4_0: return launch_cols<CoB32<false>>(s, g);
        case DT_Q8_0: return launch_cols<CoB32<true>>(s, g);
        case DT_Q4_K: return launch_cols<CoQ4K>(s, g);
        case DT_Q6_K: return m > 1 ? launch_cols<CoQ6K<Q6K_TWO_PARTS>>(s, g) : fine ? launch_cols<CoQ6K<Q6K_FINE>, true>(s, g) : launch_cols<CoQ6K<Q6K_OFFSET>, true>(s, g);
    }
    *handled = false;
    return ST_OK;
}

}  // namespace sm100
