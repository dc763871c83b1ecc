// Weight sources of the tensor-core GEMMs: how a warp fetches 16 rows x 64 weights of a quantized tensor and turns them into the
// A operand of tcgen05.mma in tensor memory.
//
// The store to tensor memory is tcgen05.st.16x256b: lane 4 g + t supplies, per step of 16 weights, the four weights 4 t .. 4 t + 3
// of rows g and g + 8.  The sum over K may run in any order, so a source gives lane t the 16 weights of a 64-weight chunk that lie
// together in memory and the activation image holds its columns in the same order (pos4 below).  A load instruction of a warp then
// touches 8 rows (8 cache lines) and not 32 as with one row per lane: the L1 looks up one line per cycle, and 32 of them per
// instruction bounded the GEMM (Q4_K, K = 4096, N = 12288, M = 1024: 299 instructions per 32 weights and lane, the load pipe 70 %
// busy).  K = 4096 before and after: Q4_K N = 12288, M = 2048 259 -> 234 us; Q8_0 N = 12288, M = 512 79 -> 74 us; Q4_0 N = 5003,
// M = 77 27.9 -> 26.2 us.
//
// Chunk c holds weights base(c) .. of a row: 64 c .. 64 c + 63 in order of K, except Q6_K, whose chunk is one 64-weight unit of the
// packed layout (sm100_layout.h).  q = index of a group of four weights in the chunk's order of K, pos4(q) = its place in the image:
// group 4 s + t belongs to step s and lane t.
#pragma once

#include "sm100_common.cuh"
#include "sm100_layout.h"

#include <cuda_bf16.h>

namespace sm100 {
namespace {

struct WeightRef {
    const uint8_t * base;
    Planes planes;       // packed layout
    int64_t row_stride;  // natural layout: bytes between rows
    int64_t blocks_per_row;
    int n;               // rows
    int last_block;      // last 32-weight block of a row
};

// 16 rows x 32 columns (the four steps of a chunk), and 16 rows x 8 columns (one step): per step [row g: two words, row g + 8: two]
__device__ __forceinline__ void tmem_st_frag4(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_frag1(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<__half2 *>(&u); }
__device__ __forceinline__ uint32_t bf2_bits(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ __nv_bfloat162 bits_bf2(uint32_t u) { return *reinterpret_cast<__nv_bfloat162 *>(&u); }
__device__ __forceinline__ float f16_bits(uint32_t h) { return __half2float(__ushort_as_half((unsigned short) h)); }
__device__ __forceinline__ uint32_t ld_u16_any(const uint8_t * p) { return __ldg((const unsigned short *) p); }

// f32 pair -> two packed bf16 pairs: hi by truncation, lo = the rest, rounded.  Truncation keeps the largest floats finite; an
// infinity leaves NaN in the rest, so a poisoned column stays non-finite.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t & hi, uint32_t & lo) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    hi = __byte_perm(ua, ub, 0x7632);
    lo = bf2_bits(__floats2bfloat162_rn(a - __uint_as_float(ua & 0xffff0000u), b - __uint_as_float(ub & 0xffff0000u)));
}
// q (two small integers, exact in bf16) times a scale d = d1 + d2 (both bf16, the rest below 2^-17 d): hi = d1 q rounded,
// d1 q - hi has at most 8 bits and is exact, lo = that + d2 q rounded once.
__device__ __forceinline__ void scale_split(uint32_t q, __nv_bfloat162 d1, __nv_bfloat162 d2, uint32_t & hi, uint32_t & lo) {
    const __nv_bfloat162 qv = bits_bf2(q);
    const __nv_bfloat162 h = __hmul2_rn(d1, qv);
    const __nv_bfloat162 r = __hfma2(d1, qv, __hneg2(h));
    hi = bf2_bits(h);
    lo = bf2_bits(__hfma2(d2, qv, r));
}
__device__ __forceinline__ void split_scale(float d, __nv_bfloat162 & d1, __nv_bfloat162 & d2) {
    const __nv_bfloat16 h = __float2bfloat16_rn(d);
    d1 = __bfloat162bfloat162(h);
    d2 = __bfloat162bfloat162(__float2bfloat16_rn(d - __bfloat162float(h)));
}

constexpr float W_PRESCALE = 256.0f;  // quantized weights of the f16 GEMM are multiplied by it before they are rounded to f16

// Interface of a source: Cursor (a lane's addresses, set up once), Regs (its share of a chunk), load() (loads only), and step<s>():
// the two words (four weights) of the lane's row `hi_row` (0: row g, 1: row g + 8) for step s, as f16 or as a bf16 split.
// prep() derives a row's scales once per chunk.

template <bool Q8, bool PACKED>
struct SrcB32 {
    static constexpr float PRESCALE = W_PRESCALE;
    struct Cursor { const uint8_t * q[2]; const uint8_t * d[2]; int off; int last; };
    struct Regs { uint32_t q[2][Q8 ? 4 : 2]; uint32_t d[2]; };
    struct ScaleF16 { __half2 d; };
    struct ScaleSplit { __nv_bfloat162 d1, d2; };
    __host__ __device__ static __forceinline__ int pos4(int q) {
        if (Q8) return 4 * (q & 3) + (q >> 2);                                            // lane t: weights 16 t + 4 s + i
        return 4 * (2 * ((q >> 2) & 1) + (q & 1)) + 2 * (q >> 3) + ((q >> 1) & 1);        // lane t: bytes 8 (t & 1) .. of block t / 2, low then high nibbles
    }
    __host__ __device__ static __forceinline__ int base(int c) { return 64 * c; }
    __host__ __device__ static __forceinline__ int k4(int q) { return 4 * q; }
    __device__ static __forceinline__ void init(Cursor & u, const WeightRef & W, const int64_t (&row)[2], int t) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (PACKED) {
                u.q[h] = W.base + row[h] * W.blocks_per_row * (Q8 ? 32 : 16) + (t & 1) * (Q8 ? 16 : 8);
                u.d[h] = W.base + W.planes.off[1] + row[h] * W.blocks_per_row * 2;
            } else {
                u.d[h] = W.base + row[h] * W.row_stride;                                   // 2-byte aligned
                u.q[h] = u.d[h] + 2 + (t & 1) * (Q8 ? 16 : 8);
            }
        }
        u.off = t >> 1;
        u.last = W.last_block;
    }
    __device__ static __forceinline__ void load(Regs & r, const Cursor & u, int c) {
        int b = 2 * c + u.off;
        const bool in = b <= u.last;   // past the end of K (a half chunk, or a whole one of the last stage): weights of scale zero
        b = in ? b : u.last;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (PACKED) {
                if constexpr (Q8) {
                    const uint4 v = __ldg((const uint4 *) (u.q[h] + (int64_t) b * 32));
                    r.q[h][0] = v.x; r.q[h][1] = v.y; r.q[h][2] = v.z; r.q[h][3] = v.w;
                } else {
                    const uint2 v = __ldg((const uint2 *) (u.q[h] + (int64_t) b * 16));
                    r.q[h][0] = v.x; r.q[h][1] = v.y;
                }
                r.d[h] = in ? ld_u16_any(u.d[h] + (int64_t) b * 2) : 0u;
            } else {
                const uint8_t * p = u.q[h] + (int64_t) b * (Q8 ? 34 : 18);
#pragma unroll
                for (int i = 0; i < (Q8 ? 4 : 2); ++i) r.q[h][i] = ld_u16_any(p + 4 * i) | ld_u16_any(p + 4 * i + 2) << 16;
                r.d[h] = in ? ld_u16_any(u.d[h] + (int64_t) b * (Q8 ? 34 : 18)) : 0u;
            }
        }
    }
    __device__ static __forceinline__ void scale(const Regs & r, int, int, int h, ScaleF16 & s) {
        s.d = __half2half2(__float2half_rn(f16_bits(r.d[h]) * W_PRESCALE));
    }
    __device__ static __forceinline__ void scale(const Regs & r, int, int, int h, ScaleSplit & s) { split_scale(f16_bits(r.d[h]), s.d1, s.d2); }
    // the step's four integers as bytes: Q8_0 signed, Q4_0 nibbles
    template <int S>
    __device__ static __forceinline__ uint32_t bytes(const Regs & r, int h) {
        if constexpr (Q8) return r.q[h][S];
        else return (S & 2 ? r.q[h][S & 1] >> 4 : r.q[h][S & 1]) & 0x0f0f0f0fu;
    }
    template <int S>
    __device__ static __forceinline__ void step(const Regs & r, int h, int, const ScaleF16 & s, uint32_t & w0, uint32_t & w1) {
        const uint32_t v = Q8 ? bytes<S>(r, h) ^ 0x80808080u : bytes<S>(r, h);
        const __half2 bias = __float2half2_rn(Q8 ? 1152.0f : 1032.0f);   // 1024 + 128 or 8
        w0 = h2_bits(__hmul2(__hsub2(bits_h2(__byte_perm(v, 0x64646464u, 0x4140u)), bias), s.d));
        w1 = h2_bits(__hmul2(__hsub2(bits_h2(__byte_perm(v, 0x64646464u, 0x4342u)), bias), s.d));
    }
    template <int S>
    __device__ static __forceinline__ void step(const Regs & r, int h, int, const ScaleSplit & s, uint32_t (&hi)[2], uint32_t (&lo)[2]) {
        const uint32_t v = bytes<S>(r, h);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t p = __byte_perm(v, 0x43434343u, i == 0 ? 0x4140u : 0x4342u);
            uint32_t q;
            if constexpr (Q8) q = bf2_bits(__hsub2(bits_bf2(p & 0xff7fff7fu), bits_bf2(p & 0xff80ff80u)));   // 128 + (b & 127) minus 128 (256 when the sign bit is set)
            else q = bf2_bits(__hsub2(bits_bf2(p), bits_bf2(0x43084308u)));                                 // 128 + nibble minus 136
            scale_split(q, s.d1, s.d2, hi[i], lo[i]);
        }
    }
};

// F16 weights: rows of K halves, 2-byte aligned at worst; used as they are, no prescale
struct SrcF16 {
    static constexpr float PRESCALE = 1.0f;
    struct Cursor { const uint8_t * p[2]; int off; int last; };
    struct Regs { uint32_t h[2][8]; };
    struct ScaleF16 {};
    __host__ __device__ static __forceinline__ int pos4(int q) { return 4 * (q & 3) + (q >> 2); }
    __device__ static __forceinline__ void init(Cursor & u, const WeightRef & W, const int64_t (&row)[2], int t) {
        for (int h = 0; h < 2; ++h) u.p[h] = W.base + row[h] * W.row_stride + (t & 1) * 32;
        u.off = t >> 1;
        u.last = W.last_block;
    }
    __device__ static __forceinline__ void load(Regs & r, const Cursor & u, int c) {
        const int b = 2 * c + u.off;
        const bool in = b <= u.last;   // past the end of K: zero (an infinity read twice would meet the zero activations)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint8_t * p = u.p[h] + (int64_t) b * 64;
            if (!in) {
#pragma unroll
                for (int i = 0; i < 8; ++i) r.h[h][i] = 0u;
            } else if ((((uintptr_t) p) & 15) == 0) {
                const uint4 a = __ldg((const uint4 *) p), e = __ldg((const uint4 *) p + 1);
                r.h[h][0] = a.x; r.h[h][1] = a.y; r.h[h][2] = a.z; r.h[h][3] = a.w;
                r.h[h][4] = e.x; r.h[h][5] = e.y; r.h[h][6] = e.z; r.h[h][7] = e.w;
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) r.h[h][i] = ld_u16_any(p + 4 * i) | ld_u16_any(p + 4 * i + 2) << 16;
            }
        }
    }
    __device__ static __forceinline__ void scale(const Regs &, int, int, int, ScaleF16 &) {}
    template <int S>
    __device__ static __forceinline__ void step(const Regs & r, int h, int, const ScaleF16 &, uint32_t & w0, uint32_t & w1) {
        w0 = r.h[h][2 * S];
        w1 = r.h[h][2 * S + 1];
    }
};

// Q4_K, packed: the tile of 16 rows x 64 weights IS lane-ordered (one 16-byte load: row g bytes 4 t .., 16 + 4 t .., then row
// g + 8), steps 0 and 1 are the low nibbles (sub-block 2 p), 2 and 3 the high ones (2 p + 1): the order of K itself.
struct SrcQ4K {
    static constexpr float PRESCALE = W_PRESCALE;
    struct Cursor { const uint8_t * q[2]; const uint8_t * h[2]; bool tile, row_major[2]; };
    struct Regs { uint32_t q[2][2]; uint4 h[2]; };
    struct ScaleF16 { __half2 d[2], m[2]; };   // per sub-block of the pair
    struct ScaleSplit { float d[2], off[2]; };
    __host__ __device__ static __forceinline__ int pos4(int q) { return q; }
    __host__ __device__ static __forceinline__ int base(int c) { return 64 * c; }
    __host__ __device__ static __forceinline__ int k4(int q) { return 4 * q; }
    __device__ static __forceinline__ void init(Cursor & u, const WeightRef & W, const int64_t (&row)[2], int t) {
        const Planes & P = W.planes;
        const int64_t full = (P.n_rows / 16) * 16;
        u.tile = row[1] < full && row[1] - row[0] == 8;   // else: rows past the last whole tile (row-major), or clamped ones
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            u.row_major[h] = row[h] >= full;
            u.q[h] = u.row_major[h] ? W.base + full * P.blocks_per_row * 128 + (row[h] - full) * P.blocks_per_row * 128 + 4 * t
                                    : W.base + (row[h] >> 4) * (P.blocks_per_row * 4) * 512 + ((row[h] & 7) * 4 + t) * 16 + ((row[h] >> 3) & 1) * 8;
            u.h[h] = W.base + P.off[1] + row[h] * P.blocks_per_row * 16;
        }
    }
    __device__ static __forceinline__ void load(Regs & r, const Cursor & u, int c) {
        if (u.tile) {
            const uint4 v = __ldg((const uint4 *) (u.q[0] + (int64_t) c * 512));
            r.q[0][0] = v.x; r.q[0][1] = v.y; r.q[1][0] = v.z; r.q[1][1] = v.w;
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint8_t * p = u.q[h] + (int64_t) c * (u.row_major[h] ? 32 : 512);
                r.q[h][0] = __ldg((const uint32_t *) p);
                r.q[h][1] = __ldg((const uint32_t *) (p + (u.row_major[h] ? 16 : 4)));
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) r.h[h] = __ldg((const uint4 *) (u.h[h] + (int64_t) (c >> 2) * 16));
    }
    // the 24-bit field of pair c & 3: sc | m << 6 of the even sub-block, then of the odd one
    __device__ static __forceinline__ uint32_t field(const uint4 & h, int c) {
        switch (c & 3) {
            case 0: return h.y;
            case 1: return __funnelshift_r(h.y, h.z, 24);
            case 2: return __funnelshift_r(h.z, h.w, 16);
            default: return h.w >> 8;
        }
    }
    __device__ static __forceinline__ void scale(const Regs & r, int c, int, int h, ScaleF16 & s) {
        const float d = f16_bits(r.h[h].x & 0xffffu) * W_PRESCALE, dmin = f16_bits(r.h[h].x >> 16) * -W_PRESCALE;
        const uint32_t f = field(r.h[h], c);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            s.d[e] = __float2half2_rn(d * (float) ((f >> (12 * e)) & 63u));
            s.m[e] = __float2half2_rn(dmin * (float) ((f >> (12 * e + 6)) & 63u));
        }
    }
    // w = D q - mn = (128 + q) D - (128 D + mn): 128 + q sits in a float's mantissa
    __device__ static __forceinline__ void scale(const Regs & r, int c, int, int h, ScaleSplit & s) {
        const float d = f16_bits(r.h[h].x & 0xffffu), dmin = f16_bits(r.h[h].x >> 16);
        const uint32_t f = field(r.h[h], c);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            s.d[e] = d * (float) ((f >> (12 * e)) & 63u);
            s.off[e] = fmaf(-128.0f, s.d[e], -(dmin * (float) ((f >> (12 * e + 6)) & 63u)));
        }
    }
    template <int S>
    __device__ static __forceinline__ uint32_t bytes(const Regs & r, int h) {
        return (S & 2 ? r.q[h][S & 1] >> 4 : r.q[h][S & 1]) & 0x0f0f0f0fu;
    }
    template <int S>
    __device__ static __forceinline__ void step(const Regs & r, int h, int, const ScaleF16 & s, uint32_t & w0, uint32_t & w1) {
        const uint32_t v = bytes<S>(r, h);
        const __half2 bias = __float2half2_rn(1024.0f);
        w0 = h2_bits(__hfma2(__hsub2(bits_h2(__byte_perm(v, 0x64646464u, 0x4140u)), bias), s.d[S >> 1], s.m[S >> 1]));
        w1 = h2_bits(__hfma2(__hsub2(bits_h2(__byte_perm(v, 0x64646464u, 0x4342u)), bias), s.d[S >> 1], s.m[S >> 1]));
    }
    template <int S>
    __device__ static __forceinline__ void step(const Regs & r, int h, int, const ScaleSplit & s, uint32_t (&hi)[2], uint32_t (&lo)[2]) {
        const uint32_t v = bytes<S>(r, h);
        const float D = s.d[S >> 1], off = s.off[S >> 1];
        split_pair(fmaf(__uint_as_float(__byte_perm(v, 0x43000000u, 0x7054)), D, off), fmaf(__uint_as_float(__byte_perm(v, 0x43000000u, 0x7154)), D, off), hi[0], lo[0]);
        split_pair(fmaf(__uint_as_float(__byte_perm(v, 0x43000000u, 0x7254)), D, off), fmaf(__uint_as_float(__byte_perm(v, 0x43000000u, 0x7354)), D, off), hi[1], lo[1]);
    }
};

// Q6_K, packed: chunk = unit u = 2 h + c of a block, lane t = its group t of 16 weights (128 h + 32 t + 16 c ..), step s = four of
// them.  Nibbles: low (t < 2) or high halves of bytes 16 (t & 1) ..; bit pairs: bits 2 t of the unit's 16 bytes.
struct SrcQ6K {
    // row g's addresses; row g + 8 lies `next` blocks on (with the eight addresses of both rows the
    // split GEMM spilled 74 bytes a thread, 12 now: us, 4096 x 32000, 8 columns 86.2 -> 75.7, 32 columns 112 -> 93; 12288 x 4096, 512 columns 166 -> 157)
    struct Cursor { const uint8_t * l; const uint8_t * x; const uint8_t * s; const uint8_t * d; int next; };
    struct Regs { uint4 n[2], b[2]; uint32_t sc[2], d[2]; };
    struct ScaleSplit { __nv_bfloat162 d1, d2; };
    __host__ __device__ static __forceinline__ int pos4(int q) { return 4 * (q & 3) + (q >> 2); }
    __host__ __device__ static __forceinline__ int base(int c) { return (c >> 2) * 256 + ((c >> 1) & 1) * 128 + (c & 1) * 16; }
    __host__ __device__ static __forceinline__ int k4(int q) { return 32 * (q >> 2) + 4 * (q & 3); }   // first weight of group q from base(c)
    __device__ static __forceinline__ void init(Cursor & u, const WeightRef & W, const int64_t (&row)[2], int t) {
        const int64_t b = row[0] * W.blocks_per_row;
        u.l = W.base + b * 128 + (t & 1) * 16;
        u.x = W.base + W.planes.off[1] + b * 64;
        u.s = W.base + W.planes.off[2] + b * 16;
        u.d = W.base + W.planes.off[3] + b * 2;
        u.next = (int) ((row[1] - row[0]) * W.blocks_per_row);
    }
    __device__ static __forceinline__ void load(Regs & r, const Cursor & u, int c) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int at = h == 0 ? c : c + 4 * u.next, block = h == 0 ? c >> 2 : (c >> 2) + u.next;
            r.n[h] = __ldg((const uint4 *) (u.l + (int64_t) at * 32));
            r.b[h] = __ldg((const uint4 *) (u.x + (int64_t) at * 16));
            r.sc[h] = __ldg((const uint32_t *) (u.s + (int64_t) at * 4));
            r.d[h] = ld_u16_any(u.d + (int64_t) block * 2);
        }
    }
    __device__ static __forceinline__ void scale(const Regs & r, int, int t, int h, ScaleSplit & s) {
        split_scale(f16_bits(r.d[h]) * (float) ((int) (r.sc[h] << (24 - 8 * t)) >> 24), s.d1, s.d2);
    }
    template <int S>
    __device__ static __forceinline__ void step(const Regs & r, int h, int t, const ScaleSplit & s, uint32_t (&hi)[2], uint32_t (&lo)[2]) {
        const uint32_t n = S == 0 ? r.n[h].x : S == 1 ? r.n[h].y : S == 2 ? r.n[h].z : r.n[h].w;
        const uint32_t b = S == 0 ? r.b[h].x : S == 1 ? r.b[h].y : S == 2 ? r.b[h].z : r.b[h].w;
        const uint32_t v = ((n >> ((t >> 1) * 4)) & 0x0f0f0f0fu) | (((b >> (2 * t)) << 4) & 0x30303030u);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            scale_split(bf2_bits(__hsub2(bits_bf2(__byte_perm(v, 0x43434343u, i == 0 ? 0x4140u : 0x4342u)), bits_bf2(0x43204320u))), s.d1, s.d2, hi[i], lo[i]);
    }
};

}  // namespace
}  // namespace sm100
