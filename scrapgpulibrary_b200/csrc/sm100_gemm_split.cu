// MUL_MAT of packed quantized weights on the fifth-generation tensor cores at the precision of the integer matvecs:
// batches of up to 32 activation columns (those that the integer column kernels serve faster stay there: q4k_columns_faster), and prompts
// of any length over Q6_K weights.
//
//   y[N, M] = W[K, N] . x[K, M]      values of src/core/ref/quant.cpp:30-108 and src/core/ref/ops.cpp:891-984
//
// The f16 GEMM (sm100_gemm.cu) rounds both operands to 11 bits (relative error 3e-4).  Here both are split into two
// bf16 numbers, w = wh + wl and x = xh + xl (16 bits of each, any magnitude a float has: no scaling, no overflow), and
//   w x = wh xh + (wh xl + wl xh)
// is three bf16 products with f32 accumulation (wl xl, below 2^-17, is taken along where it costs nothing).  The large and the small products have
// accumulators of their own (the tensor core truncates when it adds, so the long chain holds the large products only).
//
// One CTA takes 128 weight rows x TN tokens.  Warp 0 owns tensor memory and issues the MMAs; two or three groups of eight warps from warp 4 on dequantize
// the weights chunk by chunk (64 weights of each row) in packed bf16 arithmetic and store wh and wl to tensor memory, the A
// operand of the MMA.  Two ways for the activations:
//   PREP = false  (up to 32 tokens)  warps 1-3 and 20-24 read the f32 rows, split them and store the stage themselves: no launch
//                                     and no memory for it.  The padding tokens of a stage are zeroed once.
//   PREP = true   (prompts)          split_prep_x writes the stage images once per call, warps 1-3 fetch them by bulk copy.
// Few tiles, or a last wave of few, leave SMs idle: such tiles have their K range cut over several CTAs (plan_tiles), whose partial
// tiles go to scratch memory of the call; split_reduce adds them in a fixed order.
//
// What bounds it: up to 32 tokens the hand-over from chunk to chunk and the dequantizing warps (about 900 cycles a chunk of 64
// weights x 128 rows; tensor pipe 12 to 21 % busy, issue slots 53 to 66 %), with prompts the tensor core (71 % busy while a CTA is
// resident: 12 MMAs of 64 cycles in a chunk's 1090).  Measured, us, before / now: Q4_0
// 4096 x 12288, 8 columns 64 / 28; Q4_K 12288 x 4096, 24 columns 63 / 34; Q6_K 12288 x 4096, 512 columns 3740 / 157 (before: one
// launch per 8 or 4 columns).  Tried: K over a cluster with the exchange in distributed shared memory (wrong sums; taken out),
// three converting warps with their loads in registers (Q4_K, 24 columns: 41).
//
// Every wait is bounded; a CTA that gives up raises the fault flag (reported by the next stream synchronisation), drains its copies,
// frees its TMEM and returns.
#include "sm100_common.cuh"
#include "sm100_gemm_src.cuh"
#include "sm100_tc.cuh"

namespace sm100 {

bool b32_imma_serves(int64_t k);
int q4k_cols_width(int64_t k);
bool q6k_imma_serves(int64_t k);
int tail_rows(cudaStream_t s, int dtype, const void * w, int64_t k, int64_t n, int64_t row_begin, const float * x, int64_t ldx, int64_t m, float * y, int64_t ldy);

namespace {

constexpr int SP_TM = 128;             // weight rows per CTA = TMEM lanes
constexpr int SP_KC = 64;              // weights of a row per chunk
constexpr int SP_FIRST_PRODUCER = 4;
// Groups of 8 producer warps, a chunk each in turn, and the warps that bring the activations: three issue bulk copies, or eight
// convert (a lane per 8 weights of a token: with three such warps they bounded 32 columns, 1320 cycles a chunk).
template <bool PREP> constexpr int sp_groups = PREP ? 3 : 2;
template <bool PREP> constexpr int sp_threads = 32 * (SP_FIRST_PRODUCER + 8 * sp_groups<PREP> + (PREP ? 0 : 5));
constexpr int SP_BULK_WARPS = 3, SP_CONVERT_WARPS = 8;
constexpr int SP_A_COLS = 64;          // TMEM columns of a weight stage: wh (32), wl (32)
// Chunks that one CTA adds up at most.  The tensor core truncates, so the error grows with the chain: Q6_K, 512 columns, 12288 weights
// 1.68e-5, 14336 1.88e-5, 28672 3.4e-5, where the integer column kernels have 1.83e-5 at any length.
constexpr int SP_CHAIN = 208;

struct SplitArgs {
    WeightRef w;
    const float * x;           // PREP = false: activations, column stride ldx
    int64_t ldx;
    const uint8_t * image;     // PREP = true: prepared stages of all token tiles
    float * y;
    int64_t ldy;
    float * part;              // partial tiles of the cut ones: [split][tile][TN tokens][128 rows]
    int * fault;
    int n, m, k;
    int nchunks, m_tiles;
    int whole, cut, splits;    // TilePlan
};

// PREP = false: f32 activation chunks on their way, each lane's own 32 bytes per task (cp.async, read back by the same lane)
template <int TN, bool PREP>
struct SplitSmem {
    // Chunks per stage of either ring: the MMA warp's hand-over from stage to stage (about 200 cycles) shows behind the short MMAs of few
    // columns (one / two chunks, us: Q4_0 4096 x 12288, 8 columns 29.5 / 27.6; Q4_K 12288 x 4096, 24 columns 36.5 / 34.0; Q6_K 4096 x
    // 12288, 16 columns 41.4 / 39.0, 12288 x 4096, 8 columns 34.8 / 35.2).
    static constexpr int SUB = PREP ? 1 : 2;
    static constexpr int CHUNK_BYTES = 2 * TN * SP_KC * 2;              // of activations: [k / 8][xh of TN tokens, xl of TN tokens][8]
    static constexpr int B_BYTES = SUB * CHUNK_BYTES;
    static constexpr int SB = PREP ? (TN >= 128 ? 6 : 8) : 4;
    static constexpr int ACC_COLS = (TN <= 64 ? 4 : 2) * TN;
    static constexpr int SA = (512 - ACC_COLS) / (SUB * SP_A_COLS) < 6 ? (512 - ACC_COLS) / (SUB * SP_A_COLS) : 6;
    static constexpr int XS = 6;                                        // f32 chunks in flight
    uint8_t b[SB][B_BYTES];
    float4 x[PREP ? 1 : XS][2][PREP ? 1 : 32 * SP_CONVERT_WARPS];
    uint64_t full_a[SA], empty_a[SA], full_b[SB], empty_b[SB];
    uint64_t accum;
    uint32_t tmem_base;
    int abort_flag;
};

// The MMAs of a chunk.  All of one shape on an accumulator: the tensor core keeps those in order, it promises nothing for different
// shapes.  An MMA takes at least about 60 cycles, the time to read its A operand from tensor memory, whatever its columns.
//   TN <= 64: per 16-weight step two MMAs of 2 TN columns, wh [xh | xl] into D and wl [xh | xl] into the 2 TN columns behind it
//   TN = 128: three of TN columns, wh xh into D, wh xl and wl xh into the TN columns behind it
template <int TN>
__device__ __forceinline__ void mma_chunk_split(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    constexpr uint64_t B_STEP = (uint64_t) (2 * (2 * TN * 16)) >> 4, B_LOW = (uint64_t) (TN * 16) >> 4;
#pragma unroll
    for (int ks = 0; ks < SP_KC / 16; ++ks) {
        const uint32_t acc = ks == 0 ? accumulate : 1u;
        const uint64_t bh = b_desc + (uint64_t) ks * B_STEP, bl = bh + B_LOW;
        const uint32_t ah = a + 8u * ks, al = ah + 32u;
        if constexpr (TN <= 64) {
            asm volatile(
                "{\n\t.reg .pred e, pacc;\n\t"
                "elect.sync _|e, 0xffffffff;\n\t"
                "setp.ne.b32 pacc, %6, 0;\n\t"
                "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], %4, %5, pacc;\n\t"
                "@e tcgen05.mma.cta_group::1.kind::f16 [%1], [%3], %4, %5, pacc;\n\t}" ::"r"(d),
                "r"(d + 2 * TN), "r"(ah), "r"(al), "l"(bh), "r"(idesc), "r"(acc)
                : "memory");
        } else {
            asm volatile(
                "{\n\t.reg .pred e, pacc, pone;\n\t"
                "elect.sync _|e, 0xffffffff;\n\t"
                "setp.ne.b32 pacc, %7, 0;\n\t"
                "setp.eq.b32 pone, %7, %7;\n\t"
                "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], %4, %6, pacc;\n\t"
                "@e tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], %5, %6, pacc;\n\t"
                "@e tcgen05.mma.cta_group::1.kind::f16 [%1], [%3], %4, %6, pone;\n\t}" ::"r"(d),
                "r"(d + TN), "r"(ah), "r"(al), "l"(bh), "l"(bl), "r"(idesc), "r"(acc)
                : "memory");
        }
    }
}

// step ST of a warp's 16 rows: wh into the stage's columns 8 ST .., wl into 32 + 8 ST ..
template <typename S, int ST>
__device__ __forceinline__ void put_step(const typename S::Regs & r, int t, const typename S::ScaleSplit (&sc)[2], uint32_t dst) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t a[2], b[2];
        S::template step<ST>(r, h, t, sc[h], a, b);
        hi[2 * h] = a[0]; hi[2 * h + 1] = a[1];
        lo[2 * h] = b[0]; lo[2 * h + 1] = b[1];
    }
    tmem_st_frag1(dst + 8 * ST, hi);
    tmem_st_frag1(dst + 32 + 8 * ST, lo);
}

template <typename S, int TN, bool PREP>
__global__ void __launch_bounds__(sp_threads<PREP>, 1) gemm_split(const SplitArgs g) {
    using Smem = SplitSmem<TN, PREP>;
    constexpr int SUB = Smem::SUB, SA = Smem::SA, SB = Smem::SB, ACC_COLS = Smem::ACC_COLS;
    constexpr int SP_GROUPS = sp_groups<PREP>, SP_THREADS = sp_threads<PREP>, PRODUCERS = 8 * SP_GROUPS;
    constexpr int DEPTH = 2;                                             // chunks of a producer group in flight in registers
    constexpr int EPI_WARPS = TN >= 64 ? 16 : TN / 4;                    // of the first 16 producer warps
    constexpr int EPI_COLS = TN / (EPI_WARPS / 4);                       // tokens an epilogue warp reads
    static_assert(SA >= 2, "at least two weight stages");
    extern __shared__ __align__(128) uint8_t smem_raw[];
    Smem & sm = *reinterpret_cast<Smem *>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool in_part = (int) blockIdx.x >= g.whole;
    const int cut_cta = (int) blockIdx.x - g.whole;
    const int tile = in_part ? g.whole + cut_cta % g.cut : (int) blockIdx.x, split = in_part ? cut_cta / g.cut : 0, splits = in_part ? g.splits : 1;
    const int mt = tile % g.m_tiles, nt = tile / g.m_tiles;
    const int n0 = nt * SP_TM, m0 = mt * TN;
    const int m_here = g.m - m0 < TN ? g.m - m0 : TN;                    // tokens of this tile
    const int stages = g.nchunks / SUB, st_begin = (int) ((int64_t) split * stages / splits), st_count = (int) ((int64_t) (split + 1) * stages / splits) - st_begin;
    const int c_begin = st_begin * SUB, c_end = c_begin + st_count * SUB;
    volatile int * abort_flag = &sm.abort_flag;
    auto wait = [&](uint32_t bar, uint32_t parity, int site, bool patient) {
        return mbar_try_wait(bar, parity) || mbar_wait_bounded(bar, parity, abort_flag, g.fault, site, patient);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < SA; ++s) {
            mbar_init(smem_addr(&sm.full_a[s]), 8);
            mbar_init(smem_addr(&sm.empty_a[s]), 1);
        }
        for (int s = 0; s < SB; ++s) {
            mbar_init(smem_addr(&sm.full_b[s]), PREP ? 1 : (m_here + 3) / 4);   // a converting warp has four tokens
            mbar_init(smem_addr(&sm.empty_b[s]), 1);
        }
        mbar_init(smem_addr(&sm.accum), 1);
        sm.abort_flag = 0;
        fence_barrier_init();
    }
    if (!PREP) {   // padding tokens are zero for good
        for (int i = threadIdx.x; i < SB * Smem::B_BYTES / 16; i += SP_THREADS) reinterpret_cast<uint4 *>(sm.b)[i] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
    }
    if (warp == 0) {
        tmem_alloc(smem_addr(&sm.tmem_base), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *(volatile uint32_t *) &sm.tmem_base;
    const uint32_t full_a0 = smem_addr(&sm.full_a[0]), empty_a0 = smem_addr(&sm.empty_a[0]);
    const uint32_t full_b0 = smem_addr(&sm.full_b[0]), empty_b0 = smem_addr(&sm.empty_b[0]);
    const uint32_t b_smem = smem_addr(sm.b);

    if (warp >= SP_FIRST_PRODUCER && warp < SP_FIRST_PRODUCER + PRODUCERS) {
        // ---- weights (they do not depend on the predecessor on the stream): a group's eight warps take 16 rows each of a chunk
        // (a warp may write its own quarter of the TMEM lanes only: rows 32 (warp % 4) + 16 (gw / 4) ..) ----
        const int pw = warp - SP_FIRST_PRODUCER, group = pw >> 3, gw = pw & 7, t = lane & 3;
        const uint32_t lanes = (uint32_t) (32 * (warp & 3) + 16 * (gw >> 2)) << 16;
        typename S::Cursor cur;
        {
            const int64_t r0 = (int64_t) n0 + 32 * (warp & 3) + 16 * (gw >> 2) + (lane >> 2), last = g.n - 1;
            const int64_t row[2] = {r0 < last ? r0 : last, r0 + 8 < last ? r0 + 8 : last};   // rows past the tensor: clamped, never stored
            S::init(cur, g.w, row, t);
        }
        // the chunks in flight in registers: two of the group's, or the two of its stage
        static_assert(SUB == 1 || SUB == DEPTH, "the chunks of a stage are the chunks in flight");
        typename S::Regs ring[DEPTH];
        auto load = [&](typename S::Regs & r, int st, int sub) {   // past the end: a clamped, unused load
            const int c = c_begin + st * SUB + sub;
            S::load(r, cur, c < c_end ? c : c_end - 1);
        };
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) load(ring[d], SUB == 1 ? group + SP_GROUPS * d : group, SUB == 1 ? 0 : d);
        bool alive = true;
        for (int s0 = group; s0 < st_count && alive; s0 += SP_GROUPS * (SUB == 1 ? DEPTH : 1)) {
#pragma unroll
            for (int d = 0; d < DEPTH; ++d) {
                const int st = SUB == 1 ? s0 + SP_GROUPS * d : s0;
                if (st >= st_count) break;
                const int s = st % SA;
                if (SUB == 1 || d == 0) {
                    if (!__all_sync(0xffffffffu, wait(empty_a0 + 8 * s, ((uint32_t) (st / SA) & 1u) ^ 1u, 0, true))) { alive = false; break; }
                    tc_fence_after();
                }
                const int c = c_begin + st * SUB + (SUB == 1 ? 0 : d);
                const uint32_t dst = tmem + lanes + (uint32_t) (ACC_COLS + (s * SUB + (SUB == 1 ? 0 : d)) * SP_A_COLS);
                typename S::ScaleSplit sc[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) S::scale(ring[d], c, t, h, sc[h]);
                put_step<S, 0>(ring[d], t, sc, dst);
                put_step<S, 1>(ring[d], t, sc, dst);
                put_step<S, 2>(ring[d], t, sc, dst);
                put_step<S, 3>(ring[d], t, sc, dst);
                load(ring[d], SUB == 1 ? st + SP_GROUPS * DEPTH : st + SP_GROUPS, SUB == 1 ? 0 : d);
                if (SUB == 1 || d == DEPTH - 1) {
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full_a0 + 8 * s);
                }
            }
        }
        pdl_wait();
        pdl_launch_dependents();
        // ---- epilogue: lane = row, a quarter (or half, or all) of the tokens per set of four warps ----
        bool ok = alive && pw < EPI_WARPS;
        if (ok) ok = wait(smem_addr(&sm.accum), 0u, 1, true);
        if (__all_sync(0xffffffffu, ok)) {
            tc_fence_after();
            const uint32_t quarter = (uint32_t) (32 * (warp & 3)) << 16;
            const int r_in = 32 * (warp & 3) + lane, col0 = (pw >> 2) * EPI_COLS;
            const int64_t n_out = (int64_t) n0 + r_in;
#pragma unroll 1
            for (int cc = col0; cc < col0 + EPI_COLS && cc < m_here; cc += 16) {
                uint32_t a[16], b[16];
                float v[16];
                tmem_ld16(tmem + quarter + (uint32_t) cc, a);
                tmem_ld16(tmem + quarter + (uint32_t) (TN + cc), b);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(b[j]);
                if constexpr (TN <= 64) {
                    uint32_t c[16], d[16];
                    tmem_ld16(tmem + quarter + (uint32_t) (2 * TN + cc), c);
                    tmem_ld16(tmem + quarter + (uint32_t) (3 * TN + cc), d);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(c[j]) + __uint_as_float(d[j]);
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(a[j]);
                if (!in_part) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (cc + j < m_here && n_out < g.n) g.y[(int64_t) (m0 + cc + j) * g.ldy + n_out] = v[j];
                } else {
                    float * part = g.part + ((int64_t) cut_cta * TN + cc) * SP_TM + r_in;   // rows past the tensor included: the tile is whole
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (cc + j < m_here) part[j * SP_TM] = v[j];
                }
            }
        }
        __syncwarp();
    } else if (warp > 0) {
        pdl_wait();
        if (PREP) {
            if (lane == 0 && warp <= SP_BULK_WARPS) {
                const uint8_t * src = g.image + (int64_t) mt * g.nchunks * Smem::B_BYTES;
                int last = -1;
                for (int lc = warp - 1; lc < c_end - c_begin; lc += SP_BULK_WARPS) {
                    const int s = lc % SB;
                    if (!wait(empty_b0 + 8 * s, ((uint32_t) (lc / SB) & 1u) ^ 1u, 2, true)) break;
                    mbar_expect_tx(full_b0 + 8 * s, Smem::B_BYTES);
                    bulk_g2s(b_smem + s * Smem::B_BYTES, src + (int64_t) (c_begin + lc) * Smem::B_BYTES, Smem::B_BYTES, full_b0 + 8 * s);
                    last = lc;
                }
                if (*abort_flag != 0) {   // giving up: this warp's last copies land before the shared memory goes away
                    for (int lc = last; lc >= 0 && lc > last - SB; lc -= SP_BULK_WARPS) {
                        const uint32_t bar = full_b0 + 8 * (lc % SB);
                        for (uint32_t i = 0; i < (1u << 14) && !mbar_try_wait(bar, (uint32_t) (lc / SB) & 1u); ++i) __nanosleep(64);
                    }
                }
            }
        } else {
            // ---- activations: a task is 8 weights of one token (consecutive in the chunk's order of K: eight lanes read a token's
            // whole chunk), stored as two groups of four of xh and of xl ----
            constexpr int XS = Smem::XS;
            const int tid = (warp < SP_FIRST_PRODUCER ? warp - 1 : warp - SP_FIRST_PRODUCER - PRODUCERS + 3) * 32 + lane, tok = tid >> 3, j = tid & 7;
            const int kk = S::k4(2 * j), p0 = S::pos4(2 * j), p1 = S::pos4(2 * j + 1);
            const uint32_t at0 = (uint32_t) ((p0 >> 1) * (2 * TN * 16) + (p0 & 1) * 8), at1 = (uint32_t) ((p1 >> 1) * (2 * TN * 16) + (p1 & 1) * 8);
            const bool live = tok < m_here;
            const float * src = g.x + (int64_t) (live ? m0 + tok : m0) * g.ldx + kk;
            const uint32_t dst = b_smem + (uint32_t) tok * 16u, stage = smem_addr(&sm.x[0][0][tid]);
            constexpr uint32_t X_HALF = 32 * SP_CONVERT_WARPS * 16, X_BYTES = 2 * X_HALF;
            auto fetch = [&](int c) {
                if (c < c_end) {
                    const int base = S::base(c);
                    const uint32_t to = stage + (uint32_t) ((c - c_begin) % XS) * X_BYTES;
                    const bool in = live && base + kk < g.k;   // else: zero-filled
                    const float * from = in ? src + base : g.x;
                    const int bytes = in ? 16 : 0;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(from), "r"(bytes) : "memory");
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + X_HALF), "l"(from + 4), "r"(bytes) : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");   // one group per chunk, empty ones past the end
            };
            if ((tid >> 5) * 4 < m_here) {
#pragma unroll 1
                for (int i = 0; i < XS; ++i) fetch(c_begin + i);
                for (int c = c_begin; c < c_end; ++c) {
                    const int lc = c - c_begin, st = lc / SUB, s = st % SB;
                    asm volatile("cp.async.wait_group %0;" ::"n"(XS - 1) : "memory");
                    if (lc % SUB == 0 && !__all_sync(0xffffffffu, wait(empty_b0 + 8 * s, ((uint32_t) (st / SB) & 1u) ^ 1u, 2, true))) break;
                    if (live) {
                        const uint32_t from = stage + (uint32_t) (lc % XS) * X_BYTES, at = dst + (uint32_t) (s * Smem::B_BYTES + lc % SUB * Smem::CHUNK_BYTES);
                        float4 p, q;
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p.x), "=f"(p.y), "=f"(p.z), "=f"(p.w) : "r"(from) : "memory");
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w) : "r"(from + X_HALF) : "memory");
                        uint4 h, l;
                        split_pair(p.x, p.y, h.x, l.x);
                        split_pair(p.z, p.w, h.y, l.y);
                        split_pair(q.x, q.y, h.z, l.z);
                        split_pair(q.z, q.w, h.w, l.w);
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + at0), "r"(h.x), "r"(h.y) : "memory");
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + at1), "r"(h.z), "r"(h.w) : "memory");
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + at0 + TN * 16), "r"(l.x), "r"(l.y) : "memory");
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + at1 + TN * 16), "r"(l.z), "r"(l.w) : "memory");
                    }
                    if (lc % SUB == SUB - 1) {
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(full_b0 + 8 * s);
                    }
                    fetch(c + XS);
                }
                asm volatile("cp.async.wait_all;" ::: "memory");   // nothing lands after the CTA is gone
            }
        }
        __syncwarp();
    } else {
        // ---- MMA warp: the look at the next chunk's barriers is issued before this chunk's MMAs (see sm100_gemm.cu) ----
        constexpr uint32_t BF16_AB = (1u << 7) | (1u << 10);
        constexpr uint32_t IDESC = instr_desc_f16(SP_TM, TN <= 64 ? 2 * TN : TN) | BF16_AB;
        constexpr uint32_t DESC_HI = (128u >> 4) | (1u << 14);   // 128 bytes between 8-row groups; descriptor version 1
        const uint32_t b_lo0 = (b_smem >> 4) | ((uint32_t) (2 * TN * 16) >> 4) << 16;
        const int count = st_count;
        bool alive = true;
        int sa = 0, sb = 0;
        uint32_t pa = 0, pb = 0, accumulate = 0;
        uint32_t ready = (mbar_test_wait(full_b0, 0u) ? 1u : 0u) & (mbar_test_wait(full_a0, 0u) ? 1u : 0u);
        for (int lc = 0; lc < count; ++lc) {
            if (!__all_sync(0xffffffffu, ready != 0u)) {   // one answer for the warp (see sm100_gemm.cu)
                const bool ok = wait(full_b0 + 8 * sb, pb, 3, false) && wait(full_a0 + 8 * sa, pa, 4, false);
                if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
            }
            tc_fence_after();
            int sa_n = sa + 1, sb_n = sb + 1;
            uint32_t pa_n = pa, pb_n = pb;
            if (sa_n == SA) { sa_n = 0; pa_n ^= 1u; }
            if (sb_n == SB) { sb_n = 0; pb_n ^= 1u; }
            const uint32_t rb = mbar_test_wait(full_b0 + 8 * sb_n, pb_n) ? 1u : 0u;
            const uint32_t ra = mbar_test_wait(full_a0 + 8 * sa_n, pa_n) ? 1u : 0u;
            const uint64_t b_desc = ((uint64_t) DESC_HI << 32) | (b_lo0 + sb * (Smem::B_BYTES >> 4));
#pragma unroll
            for (int i = 0; i < SUB; ++i)
                mma_chunk_split<TN>(tmem, tmem + ACC_COLS + (sa * SUB + i) * SP_A_COLS, b_desc + (uint64_t) (i * (Smem::CHUNK_BYTES >> 4)), IDESC, i == 0 ? accumulate : 1u);
            accumulate = 1u;
            mma_commit2(empty_a0 + 8 * sa, empty_b0 + 8 * sb, 0u);
            ready = lc + 1 < count ? (ra & rb) : 1u;
            sa = sa_n; pa = pa_n; sb = sb_n; pb = pb_n;
        }
        __syncwarp();
        mma_commit(smem_addr(&sm.accum));
        if (!alive && lane == 0) {
            for (uint32_t i = 0; i < TC_WAIT_LIMIT && !mbar_try_wait(smem_addr(&sm.accum), 0u); ++i) __nanosleep(64);
        }
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// y of the cut tiles = sum of their parts, in the order of the splits
template <int TN>
__global__ void __launch_bounds__(256) split_reduce(const SplitArgs g) {
    pdl_wait();
    pdl_launch_dependents();
    const int64_t total = (int64_t) g.cut * (TN * SP_TM);
    for (int64_t i = (int64_t) blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t) gridDim.x * 256) {
        const int tile = g.whole + (int) (i / (TN * SP_TM)), in = (int) (i % (TN * SP_TM));
        const int row = (tile / g.m_tiles) * SP_TM + in % SP_TM, tok = (tile % g.m_tiles) * TN + in / SP_TM;
        if (row >= g.n || tok >= g.m) continue;
        float v = 0.f;
        for (int c = 0; c < g.splits; ++c) v += __ldcg(g.part + (int64_t) c * total + i);
        g.y[(int64_t) tok * g.ldy + row] = v;
    }
}

// f32 [M, K] -> stage images of Q6_K prompts: per (token tile, chunk) [k / 8][xh of TN tokens, xl of TN tokens][8], zero beyond M.
// A CTA takes TOKENS tokens x 256 weights, the four chunks of a block: a warp reads whole lines of a token, and what it makes passes through
// shared memory so that the stores are 16 TOKENS contiguous bytes too (a thread with the half chunk of a token, its loads 16 bytes of a line each: 512
// tokens of 12288, cold, 13.4 us, now 11.1; the whole product 156.7 -> 152.8, 4096 x 1024 31.2 -> 27.4).  Bound by memory.  A warp stores eight consecutive rows: with
// the rows dealt one to each warp in turn the GEMM behind it took 10 us more.
template <int TN, int TOKENS>
__global__ void __launch_bounds__(256) split_prep_x(const float * x, int64_t ldx, int m, int nchunks, uint4 * image) {
    using S = SrcQ6K;
    constexpr int ROW = TOKENS * 16 + 16;   // bytes of a row in shared memory: a unit's xh or xl of the tokens, padded against bank conflicts
    constexpr int PER = TOKENS / 8;         // tokens of a warp
    __shared__ __align__(16) uint8_t sm[64 * ROW];   // [chunk of the block][unit][xh, xl]
    pdl_wait();
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, block = blockIdx.x, tok0 = blockIdx.y * TOKENS;
    float4 v[2 * PER];   // two halves of the block per token
#pragma unroll
    for (int i = 0; i < 2 * PER; ++i) {
        const int tok = tok0 + PER * warp + (i >> 1);
        v[i] = tok < m ? __ldcg(reinterpret_cast<const float4 *>(x + (int64_t) tok * ldx + block * 256) + (i & 1) * 32 + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 2 * PER; ++i) {
        const int k = (i & 1) * 128 + 4 * lane, chunk = 2 * (k >> 7) + (k >> 4 & 1), p = S::pos4(4 * (k >> 5 & 3) + (k >> 2 & 3));   // k = base(chunk) + k4(q)
        uint2 h, l;
        split_pair(v[i].x, v[i].y, h.x, l.x);
        split_pair(v[i].z, v[i].w, h.y, l.y);
        uint8_t * at = sm + (chunk * 16 + (p >> 1) * 2) * ROW + (PER * warp + (i >> 1)) * 16 + (p & 1) * 8;
        *reinterpret_cast<uint2 *>(at) = h;
        *reinterpret_cast<uint2 *>(at + ROW) = l;
    }
    __syncthreads();
    uint4 * dst = image + ((int64_t) (tok0 / TN) * nchunks + 4 * block) * (16 * TN) + tok0 % TN;   // 16 rows of TN units per chunk
#pragma unroll
    for (int i = lane; i < 8 * TOKENS; i += 32) {   // eight rows a warp
        const int r = warp * 8 + i / TOKENS, t = i % TOKENS;
        dst[(int64_t) r * TN + t] = *reinterpret_cast<const uint4 *>(sm + r * ROW + t * 16);
    }
}

// how the tiles of g's tokens are dealt, and the memory that the partial tiles need
template <int TN, bool PREP>
TilePlan split_plan(const SplitArgs & g) {
    constexpr int SUB = SplitSmem<TN, PREP>::SUB;
    const int64_t tiles = (int64_t) ((g.n + SP_TM - 1) / SP_TM) * g.m_tiles;
    // a chunk takes 1.5 to 2 times as long as the f16 GEMM's.  The plan of a batch does not look at its columns, so that a column has the
    // same result in every batch of up to 32 columns that this kernel serves; it counts 16 (with 32 it cuts less: Q4_0 5120 x 13824, error 6.6e-6
    // against 4.9e-6, 24 columns 50.6 us against 47.4, 32 columns 51.1 against 53.3).
    return plan_tiles(tiles, g.nchunks / SUB, (TN >= 128 ? 20 : 15) * SUB, (int64_t) SP_TM * (!PREP ? 16 : g.m < TN ? g.m : TN), (g.nchunks + SP_CHAIN - 1) / SP_CHAIN);
}
template <int TN>
size_t part_bytes(const TilePlan & plan) { return (size_t) plan.cut * plan.splits * TN * SP_TM * sizeof(float); }

template <typename S, int TN, bool PREP>
int launch_split(cudaStream_t s, SplitArgs g, const TilePlan & plan, void * part) {
    g.part = (float *) part;
    g.whole = (int) plan.whole;
    g.cut = (int) plan.cut;
    g.splits = plan.splits;
    const size_t smem = sizeof(SplitSmem<TN, PREP>);
    SM100_CUDA(cudaFuncSetAttribute(gemm_split<S, TN, PREP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    int st = launch(gemm_split<S, TN, PREP>, dim3((unsigned) plan_ctas(plan)), dim3(sp_threads<PREP>), smem, s, g);
    if (st == ST_OK && plan.cut > 0) {
        const int64_t blocks = plan.cut * (TN * SP_TM / 256), cap = (int64_t) sm_count() * 8;
        st = launch(split_reduce<TN>, dim3((unsigned) (blocks < cap ? blocks : cap)), dim3(256), 0, s, g);
    }
    return st;
}

template <typename S, int TN>
int batch_split(cudaStream_t s, SplitArgs g, bool * handled) {
    TilePlan plan = split_plan<TN, false>(g);
    CallScratch mem;
    if (plan.cut > 0 && call_scratch_alloc(s, part_bytes<TN>(plan), &mem) != ST_OK) {   // no memory: one CTA per tile needs none
        if (g.nchunks > SP_CHAIN) return ST_OK;
        plan = {plan.whole + plan.cut, 0, 1, plan.cost};
    }
    *handled = true;
    const int st = launch_split<S, TN, false>(s, g, plan, mem.ptr);
    const int fr = call_scratch_free(s, mem);
    return st != ST_OK ? st : fr;
}
template <typename S>
int batch_split(cudaStream_t s, SplitArgs g, bool * handled) {
    g.m_tiles = 1;
    g.nchunks = (g.nchunks + 1) / 2 * 2;   // whole stages of two chunks
    return g.m <= 16 ? batch_split<S, 16>(s, g, handled) : batch_split<S, 32>(s, g, handled);
}

template <typename S, int TN>
int prompt_split(cudaStream_t s, SplitArgs g, const float * x, int64_t ldx, int64_t m, float * y, bool * handled) {
    // tokens per pass: the images of one pass stay below 64 MiB, and where every tile is cut its partial tiles below 256 MiB
    int64_t pass = ((int64_t) 64 << 20) / ((int64_t) g.nchunks * SP_KC * 4) / TN * TN;
    if (g.nchunks > SP_CHAIN) {
        const int64_t rows = ((int64_t) g.n + SP_TM - 1) / SP_TM * SP_TM * ((g.nchunks + SP_CHAIN - 1) / SP_CHAIN);
        const int64_t fit = ((int64_t) 256 << 20) / (rows * 4) / TN * TN;
        if (pass > fit) pass = fit;
    }
    if (pass < TN) pass = TN;
    auto tokens = [&](int64_t c0) {
        g.m = (int) (m - c0 < pass ? m - c0 : pass);
        g.m_tiles = (g.m + TN - 1) / TN;
        return split_plan<TN, true>(g);
    };
    const int64_t first = m < pass ? (m + TN - 1) / TN * TN : pass, last = (m - 1) / pass * pass;
    const size_t image_bytes = (size_t) first * g.nchunks * SP_KC * 4, part0 = part_bytes<TN>(tokens(0)), part1 = part_bytes<TN>(tokens(last));
    CallScratch mem;   // the stage images, then the partial tiles
    if (call_scratch_alloc(s, image_bytes + (part0 > part1 ? part0 : part1), &mem) != ST_OK) return ST_OK;   // no memory: the caller's column panels need none
    int st = ST_OK;
    for (int64_t c0 = 0; c0 < m && st == ST_OK; c0 += pass) {
        const TilePlan plan = tokens(c0);
        g.y = y + c0 * g.ldy;
        g.image = (const uint8_t *) mem.ptr;
        constexpr int TOKENS = TN == 64 ? 8 : 32;   // few tokens: more and shorter CTAs
        st = launch(split_prep_x<TN, TOKENS>, dim3((unsigned) (g.nchunks / 4), (unsigned) (g.m_tiles * (TN / TOKENS))), dim3(256), 0, s, x + c0 * ldx, ldx, g.m, g.nchunks, (uint4 *) mem.ptr);
        if (st == ST_OK) st = launch_split<S, TN, true>(s, g, plan, (uint8_t *) mem.ptr + image_bytes);
    }
    const int fr = call_scratch_free(s, mem);
    *handled = true;
    return st != ST_OK ? st : fr;
}

}  // namespace

// Are 9..16 columns of Q4_K faster in the integer column kernel, `width` columns a launch, than in one pass of the split GEMM?  Both times as
// measured (us, within 8 % or so over K 1024 .. 12288, N 64 .. 151936; what the rule picks was at most 5 % slower than the other way):
//   columns    a launch of 8 columns: 3.05 and, for every round of 16-row tiles (two per SM), 0.385 + 0.695 K / 1024; of a round of a narrower
//              launch 0.58 + 0.056 per column; where rows are so long that only four columns fit, 8 % more
//   split GEMM the cost of its plan times 0.031 + 0.0004 per column
// Measured, columns / split: 4096 x 12288, 9 columns 21.6 / 32.9, 16 columns 26.9 / 35.6; 4096 x 4096, 16 columns 13.0 / 15.3; 4096 x 1024,
// 16 columns 11.7 / 9.4; 12288 x 4096, 12 columns 31.4 / 30.9.  The line is drawn at 16 columns because the split GEMM is the more accurate way (error
// 7e-6; 4e-5 to 1e-4 with the column kernel): beyond, and for 8 columns of Q6_K, the column kernels win little and seldom (Q4_K 5120 x 13824,
// 17 columns 43.4 / 49.7, 24 columns 49.4 / 51.4, 4096 x 4096, 17 columns 16.9 / 15.7; Q6_K 5120 x 13824, 8 columns 47.0 / 48.5, 4096 x 4096 17.2 / 15.0).
bool q4k_columns_faster(int64_t k, int64_t n, int64_t m, int width) {
    if (m > 16) return false;
    const int chunks = (int) ((k + 2 * SP_KC - 1) / (2 * SP_KC)) * 2;
    const double cost = (double) plan_tiles((n / 16 * 16 + SP_TM - 1) / SP_TM, chunks / 2, 30, SP_TM * 32, (chunks + SP_CHAIN - 1) / SP_CHAIN).cost, kk = (double) k / 1024;
    const int64_t at_once = 2 * (int64_t) sm_count(), rounds = (n / 16 + at_once - 1) / at_once;
    double columns = 0;
    for (int64_t c = 0; c < m; c += width) {
        const int64_t mm = m - c < width ? m - c : width;
        columns += 3.05 + (double) rounds * (0.385 + 0.695 * kk) * (mm == 8 ? 1.0 : 0.58 + 0.056 * (double) mm);
    }
    return columns * (width == 8 ? 1.0 : 1.08) < cost * (0.031 + 0.0004 * (double) m);
}

// Packed Q4_0 / Q8_0 / Q4_K / Q6_K with up to 32 columns, or Q6_K with any number; *handled = false (and ST_OK) when the shape is
// left to the caller's other kernels.
// It takes the place of the integer column kernels only, whose 16-bit activations are coarser than its operands (relative error
// 2e-5 to 6e-5; 5e-6 to 2e-5 here).  What those leave to the f32 kernels (2e-7) stays in f32: tensors of fewer than 16 rows, the
// last N mod 16 rows (a launch of their own behind the GEMM's: 3 to 8 us up to 64 columns, 26 for 512), rows that are not whole units
// or too long for them.
int gemm_split_mul_mat(cudaStream_t s, int dtype, const void * w, int64_t k, int64_t n, const float * x, int64_t ldx, int64_t m, float * y, int64_t ldy,
                       bool * handled) {
    *handled = false;
    if (n < 16 || k <= 0 || (m > 32 && dtype != DT_Q6_K)) return ST_OK;
    switch (dtype) {
        case DT_Q4_0: case DT_Q8_0: if (!b32_imma_serves(k)) return ST_OK; break;
        case DT_Q4_K: if (q4k_cols_width(k) == 0) return ST_OK; break;
        case DT_Q6_K: if (!q6k_imma_serves(k)) return ST_OK; break;
        default: return ST_OK;
    }
    if (n > INT32_MAX - SP_TM || m > INT32_MAX / 2) return ST_OK;
    if ((((uintptr_t) x) & 15) != 0 || (m > 1 && ldx % 4 != 0) || (((uintptr_t) w) & 31) != 0) return ST_OK;
    const int64_t full = n / 16 * 16;
    SplitArgs g = {};
    const int fw = fault_word(FAULT_SPLIT, &g.fault);
    if (fw != ST_OK) return fw;
    g.w.base = (const uint8_t *) w;
    g.w.planes = planes_for(dtype, n, k);
    g.w.blocks_per_row = k / block_elems(dtype);
    g.w.n = (int) n;
    g.w.last_block = (int) (k / 32) - 1;
    g.x = x;
    g.ldx = ldx;
    g.y = y;
    g.ldy = ldy;
    g.n = (int) full;
    g.m = (int) m;
    g.k = (int) k;
    g.nchunks = (int) ((k + SP_KC - 1) / SP_KC);
    int st = ST_OK;
    if (m > 32) {
        st = m <= 64 ? prompt_split<SrcQ6K, 64>(s, g, x, ldx, m, y, handled) : prompt_split<SrcQ6K, 128>(s, g, x, ldx, m, y, handled);
    } else {
        switch (dtype) {
            case DT_Q4_0: st = batch_split<SrcB32<false, true>>(s, g, handled); break;
            case DT_Q8_0: st = batch_split<SrcB32<true, true>>(s, g, handled); break;
            case DT_Q4_K: st = batch_split<SrcQ4K>(s, g, handled); break;
            default: st = batch_split<SrcQ6K>(s, g, handled); break;
        }
    }
    if (st != ST_OK || !*handled) return st;
    if (full < n) st = tail_rows(s, dtype, w, k, n, full, x, ldx, m, y, ldy);
    *handled = st == ST_OK;
    return st;
}

}  // namespace sm100
