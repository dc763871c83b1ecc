// Prefill MUL_MAT (33 activation columns and more) on the fifth-generation tensor cores.
//
//   y[N, M] = W[K, N] . x[K, M]      W quantized (Q8_0, Q4_0, Q4_K) or F16, x and y f32
//
// replaces the reference's tiled GEMM (src/backends/opencl11/kernels/mul_mm.cl:271, dispatched from
// src/backends/opencl11/opencl_api.cpp for batches above the matvec limit) and has to agree with the CPU
// reference (src/core/ref/ops.cpp:891-984) to NMSE <= 1e-6.
//
// Two launches per call:
//
//  1. gemm_prep_x   converts the activations to f16 once, normalised per token by a power of two (so the
//                   largest element of a token sits in [8192, 16384) whatever its magnitude), and writes
//                   them in the shared-memory image the tensor core wants: per (token tile, 64-wide K chunk)
//                   one contiguous block of 8-token x 16-byte core matrices.  A consumer CTA then fetches a
//                   whole B stage with one bulk copy (cp.async.bulk, completion on an mbarrier).
//
//  2. gemm_tc       one CTA per 128 weight rows x TN tokens (TN = 128 or 256).  Warp 0 owns the tensor memory
//                   and issues tcgen05.mma (kind::f16, 128 x TN x 16 per instruction, f32 accumulator of TN
//                   TMEM columns), warps 1-3 issue the bulk copies of the B stages in turn (a warp gets one
//                   bulk copy through per ~530 cycles), warps 4-27 dequantize the CTA's weight rows chunk by
//                   chunk to f16 (weights are multiplied by 256 to keep small scales out of the f16
//                   subnormals) straight into tensor memory with tcgen05.st, from where the MMA reads its A
//                   operand, so that shared memory carries the activations only (sm100_gemm_src.cuh).
//                   Weight stages and activation stages are two rings with their own full/empty
//                   mbarriers; tcgen05.commit hands both back.  When the last commit lands, warps 4-19 read
//                   the accumulator with tcgen05.ld, undo the two scalings and store y.
//
// f16 operands with f32 accumulation: each product carries two roundings of 2^-11 relative size, which
// puts the NMSE near 2e-7.  Every wait on an mbarrier is bounded; a CTA that gives up raises a fault flag
// (reported by the next stream synchronisation), drains its copies, frees its TMEM and returns.
#include "sm100_common.cuh"
#include "sm100_gemm_src.cuh"
#include "sm100_tc.cuh"

#include <cstdlib>
#include <mutex>
#include <vector>

namespace sm100 {

int device_scratch(int slot, size_t bytes, void ** out);

namespace {

constexpr int TM = 128;            // weight rows per CTA = rows of one tcgen05.mma = TMEM lanes
// Warp roles.  The MMA warp is warp 0: as a young warp it was starved by the polling producers (each of its
// instructions took 50-80 cycles to issue).
constexpr int WARP_MMA = 0;        // owns TMEM and issues the MMAs
constexpr int WARP_BULK = 1;       // warps 1-3 issue the bulk copies of the activation stages, a chunk each in turn
constexpr int BULK_WARPS = 3;
constexpr int FIRST_PRODUCER = 4;  // warps 4.. dequantize; the first 16 of them then run the epilogue
// Producer warps: 8 warps = 256 (row, 32-weight block) tasks = one 64-wide chunk of the 128 rows, so 24 warps are three
// groups that take the chunks in turn.  A producer's instruction stream is a dependent chain (~7 cycles per
// instruction), so the third group buys throughput that the issue slots still have.
constexpr int PRODUCER_WARPS = 24;
constexpr int EPILOGUE_WARPS = 16;
constexpr int GEMM_THREADS = 32 * (FIRST_PRODUCER + PRODUCER_WARPS);

// ---------------------------------------------------------------------------------------------
// Shared memory of one CTA
// ---------------------------------------------------------------------------------------------
constexpr int KC = 64;   // weights of a row per chunk

// SUB chunks make a stage of either ring: the MMA warp's hand-over from stage to stage costs about 200 cycles, which four MMAs of 128
// columns (256 cycles) do not hide.
template <int TN, int STAGES, int SUB>
struct GemmSmem {
    static constexpr int CHUNK_BYTES = TN * KC * 2;
    static constexpr int B_BYTES = SUB * CHUNK_BYTES;
    // Weight stages: as many as the tensor memory columns left by the accumulator hold, at most 8.  The two rings have
    // their own barriers: the activation copies are the long-latency side (~2 us under load) and want every byte of shared
    // memory in flight.
    static constexpr int SA = (512 - TN) / (SUB * (KC / 2)) < 8 ? (512 - TN) / (SUB * (KC / 2)) : 8;
    uint8_t b[STAGES][B_BYTES];  // [k / 8][token][8 halves]
    uint64_t full_a[SA];         // producers -> MMA: one arrival per producer warp of a group
    uint64_t empty_a[SA];        // MMA commit -> producers
    uint64_t full_b[STAGES];     // bulk copy -> MMA: the issuing lane's expect_tx arrival + the bytes
    uint64_t empty_b[STAGES];    // MMA commit -> bulk warp
    uint64_t accum;              // last commit -> epilogue
    uint32_t tmem_base;
    int abort_flag;
};

struct GemmArgs {
    WeightRef w;
    const __half * xh;       // prepared activations of this pass
    const float * tokscale;  // per token: 1 / token scale
    float out_scale;         // 1 / weight prescale
    float * y;
    int64_t ldy;
    int * fault;
    int n, m;      // weight rows; tokens of this pass
    int nchunks;   // ceil(K / KC), a whole number of stages
    int m_tiles;
};

// The dequantized weights go to tensor memory (tcgen05.st by the producers, A operand of the MMA read from TMEM), so that
// shared memory carries only the activation stages.  TMEM columns: the accumulator of TN, then per chunk of a stage KC / 2 columns of A
// (two f16 per column).
template <typename S, int TN, int STAGES, int SUB>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_tc(const GemmArgs g) {
    constexpr int GROUP_WARPS = 8;                          // a chunk of 128 rows: eight warps of 16 rows each
    constexpr int GROUPS = PRODUCER_WARPS / GROUP_WARPS;    // groups take the chunks in turn
    extern __shared__ __align__(128) uint8_t smem_raw[];
    using Smem = GemmSmem<TN, STAGES, SUB>;
    constexpr int ACC_COLS = TN;
    constexpr int A_COLS = SUB * KC / 2;                             // per stage
    constexpr int SA = Smem::SA;
    static_assert(SA >= 2, "at least two weight stages");
    constexpr int USED_COLS = ACC_COLS + SA * A_COLS;
    constexpr int TMEM_COLS = USED_COLS <= 32 ? 32 : USED_COLS <= 64 ? 64 : USED_COLS <= 128 ? 128 : USED_COLS <= 256 ? 256 : 512;
    static_assert(USED_COLS <= 512, "accumulator and weight stages exceed the tensor memory");
    Smem & sm = *reinterpret_cast<Smem *>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x % g.m_tiles, nt = blockIdx.x / g.m_tiles;
    const int n0 = nt * TM, m0 = mt * TN;
    volatile int * abort_flag = &sm.abort_flag;

    if (threadIdx.x == 0) {
        for (int s = 0; s < SA; ++s) {
            mbar_init(smem_addr(&sm.full_a[s]), GROUP_WARPS);
            mbar_init(smem_addr(&sm.empty_a[s]), 1);
        }
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_addr(&sm.full_b[s]), 1);
            mbar_init(smem_addr(&sm.empty_b[s]), 1);
        }
        mbar_init(smem_addr(&sm.accum), 1);
        sm.abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == WARP_MMA) {
        tmem_alloc(smem_addr(&sm.tmem_base), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *(volatile uint32_t *) &sm.tmem_base;
    // barrier addresses advance by 8 bytes per stage, operand stages by their byte size
    const uint32_t full_a0 = smem_addr(&sm.full_a[0]), empty_a0 = smem_addr(&sm.empty_a[0]);
    const uint32_t full_b0 = smem_addr(&sm.full_b[0]), empty_b0 = smem_addr(&sm.empty_b[0]);
    const uint32_t b_smem = smem_addr(sm.b[0]);

    // Everything above, and the weight side below, overlaps the activation preparation that precedes this kernel
    // in the stream: only the bulk-copy warp (prepared activations) and the epilogue (token factors, output) wait
    // for it.  That kernel itself starts only after everything before it has completed, so nothing older is in flight.

    if (warp >= FIRST_PRODUCER) {
        // ---- A operand.  A group's eight warps take 16 rows each of a chunk (a warp may only write its own quarter of the TMEM
        // lanes: rows 32 (warp % 4) + 16 (gw / 4) ..); lane 4 g + t holds 16 weights of rows g and g + 8 (sm100_gemm_src.cuh).
        // DEPTH of the group's chunks are kept in flight in registers to cover the L2/HBM latency.
        constexpr int DEPTH = 2;
        static_assert(SUB == 1 || SUB == DEPTH, "the chunks of a stage are the chunks in flight");
        const int pw = warp - FIRST_PRODUCER;
        const int group = pw / GROUP_WARPS, gw = pw % GROUP_WARPS, t = lane & 3;
        const int row_in = 32 * (warp & 3) + 16 * (gw >> 2);
        // Group g takes the stages g, g + GROUPS, ...  Rows past the tensor are clamped to the last one: such rows are never stored.
        // With two chunks a stage these are the chunks in flight.
        const int units = g.nchunks / SUB;
        typename S::Cursor cur;
        {
            const int64_t r0 = (int64_t) n0 + row_in + (lane >> 2), last = g.n - 1;
            const int64_t row[2] = {r0 < last ? r0 : last, r0 + 8 < last ? r0 + 8 : last};
            S::init(cur, g.w, row, t);
        }
        auto load = [&](typename S::Regs & r, int st, int sub) {   // past the end: a clamped, unused load
            S::load(r, cur, (st < units ? st : units - 1) * SUB + sub);
        };
        // one chunk of the warp's 16 rows to tensor memory
        auto put = [&](const typename S::Regs & r, int chunk, uint32_t dst) {
            uint32_t out[16];   // per step: row g two words, row g + 8 two words
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                typename S::ScaleF16 sc;
                S::scale(r, chunk, t, h, sc);
                S::template step<0>(r, h, t, sc, out[2 * h], out[2 * h + 1]);
                S::template step<1>(r, h, t, sc, out[4 + 2 * h], out[4 + 2 * h + 1]);
                S::template step<2>(r, h, t, sc, out[8 + 2 * h], out[8 + 2 * h + 1]);
                S::template step<3>(r, h, t, sc, out[12 + 2 * h], out[12 + 2 * h + 1]);
            }
            tmem_st_frag4(dst, out);
        };
        const uint32_t dst0 = tmem + ((uint32_t) row_in << 16) + (uint32_t) ACC_COLS;
        typename S::Regs ring[DEPTH];
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) load(ring[d], SUB == 1 ? group + GROUPS * d : group, SUB == 1 ? 0 : d);
        bool alive = true;
        for (int u0 = group; u0 < units && alive; u0 += GROUPS * (SUB == 1 ? DEPTH : 1)) {
#pragma unroll
            for (int d = 0; d < DEPTH; ++d) {
                const int st = SUB == 1 ? u0 + GROUPS * d : u0;
                if (st >= units) break;
                const int s = st % SA;
                if (SUB == 1 || d == 0) {   // the stage is free once the MMAs that used it last have retired
                    const uint32_t phase = (uint32_t) (st / SA) & 1u;
                    bool ok = mbar_try_wait(empty_a0 + 8 * s, phase ^ 1u);
                    if (!ok) ok = mbar_wait_bounded(empty_a0 + 8 * s, phase ^ 1u, abort_flag, g.fault, 0, true);
                    if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
                    tc_fence_after();   // those MMAs (observed through the barrier) precede these stores
                }
                put(ring[d], SUB == 1 ? st : st * SUB + d, dst0 + (uint32_t) (s * A_COLS + (SUB == 1 ? 0 : d * (KC / 2))));
                load(ring[d], SUB == 1 ? st + GROUPS * DEPTH : st + GROUPS, SUB == 1 ? 0 : d);
                if (SUB == 1 || d == DEPTH - 1) {
                    tmem_st_wait();
                    tc_fence_before();   // the stores are ordered before the MMAs that the arrival releases
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full_a0 + 8 * s);
                }
            }
        }
        // the dependency wait (long satisfied: the activations have been flowing) comes before the successor is
        // released, as in every kernel of this library: a successor's early section then overlaps this kernel only
        pdl_wait();
        pdl_launch_dependents();

        // ---- epilogue: a warp may read the TMEM lanes 32 (warp % 4) ..; four consecutive producer warps cover
        // the four lane quarters, and each such set takes a quarter of the columns ----
        bool acc_ok = alive;
        if (acc_ok) {
            acc_ok = mbar_try_wait(smem_addr(&sm.accum), 0u);
            if (!acc_ok) acc_ok = mbar_wait_bounded(smem_addr(&sm.accum), 0u, abort_flag, g.fault, 1, true);
        }
        if (__all_sync(0xffffffffu, acc_ok) && pw < EPILOGUE_WARPS) {
            tc_fence_after();
            const int lane_base = 32 * (warp & 3);
            const int col_base = (pw >> 2) * (TN / 4);
            const int64_t n_out = (int64_t) n0 + lane_base + lane;
#pragma unroll 1
            for (int cc = 0; cc < TN / 4; cc += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + ((uint32_t) lane_base << 16) + (uint32_t) (col_base + cc), r);
                // the token factors are fetched before any store: a load after a store to memory that may alias
                // is not moved up by the compiler, and 16 dependent trips to L2 per pass cost ~5 us per CTA
                float f[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) f[j] = __ldcg(g.tokscale + m0 + col_base + cc + j) * g.out_scale;   // allocated for whole tiles
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int tok = m0 + col_base + cc + j;
                    if (tok < g.m && n_out < g.n) g.y[(int64_t) tok * g.ldy + n_out] = __uint_as_float(r[j]) * f[j];
                }
            }
        }
    } else if (warp >= WARP_BULK) {
        // ---- B operand: one bulk copy per stage, issued as soon as the stage is free.  A warp gets one bulk copy
        // through per ~530 cycles whatever its size (measured: 16 KB copies from one thread 31 B/cycle, from four
        // warps 113 B/cycle), so the chunks go round BULK_WARPS issuing warps. ----
        if (lane == 0) {
            pdl_wait();
            const uint8_t * src = reinterpret_cast<const uint8_t *>(g.xh) + (int64_t) mt * g.nchunks * Smem::CHUNK_BYTES;
            int last = -1;
            for (int c = warp - WARP_BULK; c < g.nchunks / SUB; c += BULK_WARPS) {
                const int s = c % STAGES;
                const uint32_t phase = (uint32_t) (c / STAGES) & 1u;
                if (!mbar_try_wait(empty_b0 + 8 * s, phase ^ 1u) && !mbar_wait_bounded(empty_b0 + 8 * s, phase ^ 1u, abort_flag, g.fault, 2, true)) break;
                mbar_expect_tx(full_b0 + 8 * s, Smem::B_BYTES);
                bulk_g2s(b_smem + s * Smem::B_BYTES, src + (int64_t) c * Smem::B_BYTES, Smem::B_BYTES, full_b0 + 8 * s);
                last = c;
            }
            // Every copy has landed once the MMA warp has passed its stage's barrier, which it does for every chunk
            // before the CTA ends.  Only a CTA that is giving up can have copies in flight when it leaves: wait,
            // briefly, for this warp's last ones so that they do not land in freed shared memory.
            if (*abort_flag != 0) {
                for (int c = last; c >= 0 && c > last - STAGES; c -= BULK_WARPS) {
                    const uint32_t bar = full_b0 + 8 * (c % STAGES);
                    for (uint32_t i = 0; i < (1u << 14) && !mbar_try_wait(bar, (uint32_t) (c / STAGES) & 1u); ++i) __nanosleep(64);
                }
            }
        }
        __syncwarp();
    } else {
        // ---- MMA warp (warp 0).  This loop is one warp's serial instruction stream and bounds the kernel,
        // so it is kept lean: one barrier per stage, descriptors are a base plus compile-time offsets in
        // their low word, stage and phase are counters. ----
        constexpr uint32_t IDESC = instr_desc_f16(TM, TN);
        constexpr uint32_t DESC_HI = (128u >> 4) | (1u << 14);  // 128 bytes between 8-row groups; descriptor version 1
        const uint32_t b_lo0 = (b_smem >> 4) | ((uint32_t) (TN * 16) >> 4) << 16;
        bool alive = true;
        const uint32_t issuer = lane == 0 ? 1u : 0u;   // the lane that issues the MMAs and the commits (always the same one)
        int sa = 0, sb = 0;                       // stage of the weight ring and of the activation ring
        uint32_t pa = 0, pb = 0, accumulate = 0;
        // Both rings run several stages ahead, so the barriers of a chunk are almost always complete when this warp
        // gets to it - but asking costs a round trip (~250 cycles per barrier for this lone warp, two thirds of
        // the loop).  The look at chunk c + 1's barriers is therefore issued before chunk c's MMAs and its answer
        // used an iteration later; only a "not yet" takes the waiting path.
        uint32_t ready = (mbar_test_wait(full_b0, 0u) ? 1u : 0u) & (mbar_test_wait(full_a0, 0u) ? 1u : 0u);
        const int stages = g.nchunks / SUB;
        for (int c = 0; c < stages; ++c) {
            if (!__all_sync(0xffffffffu, ready != 0u)) {   // one answer for the warp: a lane may have looked before a phase completed, another after
                bool ok = mbar_try_wait(full_b0 + 8 * sb, pb);
                if (!ok) ok = mbar_wait_bounded(full_b0 + 8 * sb, pb, abort_flag, g.fault, 3, false);
                if (ok) {
                    ok = mbar_try_wait(full_a0 + 8 * sa, pa);
                    if (!ok) ok = mbar_wait_bounded(full_a0 + 8 * sa, pa, abort_flag, g.fault, 4, false);
                }
                if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
            }
            tc_fence_after();
            // next chunk's stages
            int sa_n = sa + 1, sb_n = sb + 1;
            uint32_t pa_n = pa, pb_n = pb;
            if (sa_n == SA) { sa_n = 0; pa_n ^= 1u; }
            if (sb_n == STAGES) { sb_n = 0; pb_n ^= 1u; }
            const uint32_t rb = mbar_test_wait(full_b0 + 8 * sb_n, pb_n) ? 1u : 0u;   // read after this chunk's MMAs are issued
            const uint32_t ra = mbar_test_wait(full_a0 + 8 * sa_n, pa_n) ? 1u : 0u;
            const uint64_t b_desc = ((uint64_t) DESC_HI << 32) | (b_lo0 + sb * (Smem::B_BYTES >> 4));
#pragma unroll
            for (int i = 0; i < SUB; ++i)   // chunks of the stage
                mma4_f16_ta(tmem, tmem + ACC_COLS + sa * A_COLS + i * (KC / 2), b_desc + (uint64_t) (i * (Smem::CHUNK_BYTES >> 4)), (uint64_t) (2 * TN * 16 >> 4), IDESC,
                            i == 0 ? accumulate : 1u, issuer);
            accumulate = 1u;
            mma_commit2(empty_a0 + 8 * sa, empty_b0 + 8 * sb, issuer);   // each commit covers every MMA issued so far
            ready = c + 1 < stages ? (ra & rb) : 1u;
            sa = sa_n; pa = pa_n; sb = sb_n; pb = pb_n;
        }
        __syncwarp();
        // the accumulator is complete (or abandoned) once everything issued so far has retired
        mma_commit(smem_addr(&sm.accum));
        if (!alive && lane == 0) {
            for (uint32_t i = 0; i < TC_WAIT_LIMIT && !mbar_try_wait(smem_addr(&sm.accum), 0u); ++i) __nanosleep(64);
        }
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == WARP_MMA) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------------------------
// Activation preparation: f32 [M, K] (column stride ldx) -> normalised f16 stage images + token factors
// ---------------------------------------------------------------------------------------------
// A CTA takes `toks` consecutive tokens (a power of two, 1..8) with 256 / toks threads each and keeps their rows in
// registers (up to V float4 per thread, all requested at once): one trip to memory gives both the
// token's largest magnitude and, after the scale is known, the f16 image.  Rows too long for the registers
// (K > 32768) take the two-pass path: the same loop twice.
// What bounds it is the number of CTAs and of bytes in flight: few float4 a thread (V = 4 up to K = 4096) and so many CTAs, of few registers each, rather than
// eight tokens a CTA with 32 float4 a thread.  Products of 77 tokens (Q4_0, 4096 x 5003):
// 23.2 -> 21.1 us behind one another (inputs that no cache holds: no gain), of 512 (Q8_0, 4096 x 12288) no more than repeated timing differs by; the preparation alone, cold,
// 6.5 -> 4.1 and 8.0 -> 6.0.
constexpr int PREP_MAX_V = 32;

// `order`: places of the groups of four weights in a chunk (pos4 of the weight source): 0 = in order of K, 1 = as Q8_0 and F16
// weights want them, 2 = Q4_0.
template <int TN, int V>
__global__ void __launch_bounds__(256) gemm_prep_x(const float * x, int64_t ldx, int m, int k, int nchunks, int toks, int order, float * tokscale,
                                                   __half * xh) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float s_amax[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tpt = 256 / toks;                  // threads per token: 32, 64, 128 or 256
    const int tok = blockIdx.x * toks + threadIdx.x / tpt;
    const int r = threadIdx.x % tpt;
    const int kpad4 = nchunks * (KC / 4);        // float4 per token in the image (K padded to whole chunks)
    const int k4 = k / 4;
    const bool in_regs = kpad4 <= V * tpt;
    const float4 * row = reinterpret_cast<const float4 *>(x + (int64_t) tok * ldx);
    const bool tok_ok = tok < m;
    float4 v[V];
    float amax = 0.0f;
    if (in_regs) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const int idx = r + i * tpt;
            v[i] = tok_ok && idx < k4 ? __ldcg(row + idx) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < V; ++i)
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
    } else if (tok_ok) {
#pragma unroll 8
        for (int idx = r; idx < k4; idx += tpt) {
            const float4 t = __ldcg(row + idx);
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(t.x), fabsf(t.y)), fmaxf(fabsf(t.z), fabsf(t.w))));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) s_amax[warp] = amax;
    __syncthreads();
    const int wpt = tpt / 32, w0 = (threadIdx.x / tpt) * wpt;   // the token's warps
    amax = 0.0f;
    for (int w = 0; w < wpt; ++w) amax = fmaxf(amax, s_amax[w0 + w]);
    int sh = 0;
    if (amax > 0.0f && amax <= 3.0e38f) {
        sh = 13 - ilogbf(amax);
        sh = sh > 100 ? 100 : sh < -100 ? -100 : sh;
    }
    const float scale = ldexpf(1.0f, sh);
    if (r == 0) tokscale[tok] = ldexpf(1.0f, -sh);
    // image: [token tile][chunk][k / 8][token in tile][8 halves]; a float4 is half of one 16-byte unit
    const int mt = tok / TN, tt = tok % TN;
    __half * img = xh + (int64_t) mt * nchunks * (TN * KC) + tt * 8;
    auto put = [&](int idx, const float4 & t) {
        const int c = idx / (KC / 4), q = idx % (KC / 4);
        const int p = order == 0 ? q : order == 1 ? SrcF16::pos4(q) : SrcB32<false, true>::pos4(q);
        const __half2 h0 = __floats2half2_rn(t.x * scale, t.y * scale), h1 = __floats2half2_rn(t.z * scale, t.w * scale);
        *reinterpret_cast<uint2 *>(img + (int64_t) c * (TN * KC) + (p >> 1) * (TN * 8) + (p & 1) * 4) = make_uint2(h2_bits(h0), h2_bits(h1));
    };
    if (in_regs) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
            const int idx = r + i * tpt;
            if (idx < kpad4) put(idx, v[i]);
        }
    } else {
#pragma unroll 8
        for (int idx = r; idx < kpad4; idx += tpt) put(idx, tok_ok && idx < k4 ? __ldcg(row + idx) : make_float4(0.f, 0.f, 0.f, 0.f));
    }
}

template <typename S, int TN, int STAGES, int SUB>
int launch_gemm(cudaStream_t s, GemmArgs g, int n_tiles) {
    g.out_scale = 1.0f / S::PRESCALE;
    using Smem = GemmSmem<TN, STAGES, SUB>;
    static std::mutex mu;
    static std::vector<char> configured;
    int dev = 0;
    SM100_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lock(mu);
        if ((int) configured.size() <= dev) configured.resize(dev + 1, 0);
        if (!configured[dev]) {
            SM100_CUDA(cudaFuncSetAttribute(gemm_tc<S, TN, STAGES, SUB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(Smem)));
            configured[dev] = 1;
        }
    }
    return launch(gemm_tc<S, TN, STAGES, SUB>, dim3((unsigned) (n_tiles * g.m_tiles)), dim3(GEMM_THREADS), sizeof(Smem), s, g);
}

template <int TN, int STAGES, int SUB>
int launch_gemm_dtype(cudaStream_t s, int dtype, int layout, const GemmArgs & g, int n_tiles) {
    const bool packed = layout == LAYOUT_PACKED;
    switch (dtype) {
        case DT_Q8_0:
            return packed ? launch_gemm<SrcB32<true, true>, TN, STAGES, SUB>(s, g, n_tiles) : launch_gemm<SrcB32<true, false>, TN, STAGES, SUB>(s, g, n_tiles);
        case DT_Q4_0:
            return packed ? launch_gemm<SrcB32<false, true>, TN, STAGES, SUB>(s, g, n_tiles) : launch_gemm<SrcB32<false, false>, TN, STAGES, SUB>(s, g, n_tiles);
        case DT_Q4_K: return launch_gemm<SrcQ4K, TN, STAGES, SUB>(s, g, n_tiles);
        case DT_F16: return launch_gemm<SrcF16, TN, STAGES, SUB>(s, g, n_tiles);
    }
    return fail(ST_UNSUPPORTED, "gemm: no tensor-core source for dtype %d", dtype);
}

template <int TN, int STAGES, int SUB>
int gemm_passes(cudaStream_t s, int dtype, int layout, GemmArgs g, const float * x, int64_t ldx, int64_t m, int64_t k, float * y) {
    const int n_tiles = (g.n + TM - 1) / TM;
    g.nchunks = (int) ((k + SUB * KC - 1) / (SUB * KC)) * SUB;
    // tokens per pass: the prepared activations of one pass stay below 64 MiB
    int64_t pass = ((int64_t) 64 << 20) / ((int64_t) g.nchunks * KC * 2) / TN * TN;
    if (pass < TN) pass = TN;
    for (int64_t c0 = 0; c0 < m; c0 += pass) {
        const int64_t mm = m - c0 < pass ? m - c0 : pass;
        const int m_tiles = (int) ((mm + TN - 1) / TN);
        const int64_t mpad = (int64_t) m_tiles * TN;
        const size_t scale_bytes = ((size_t) mpad * sizeof(float) + 255) / 256 * 256;
        const size_t bytes = scale_bytes + (size_t) mpad * g.nchunks * KC * sizeof(__half);
        void * ws = nullptr;
        int st = device_scratch(1, bytes, &ws);
        if (st != ST_OK) return st;
        float * tokscale = (float *) ws;
        __half * xh = (__half *) ((uint8_t *) ws + scale_bytes);
        // Tokens per CTA: one where the GEMM fills the SMs, so that the preparation has many CTAs.  Else as many (up to 8, and to 32 float4 a thread) as leave
        // the GEMM's CTAs, which share an SM with nobody, the SMs that they start on meanwhile (Q4_0 2304 x 10688, 46 tokens, 84 CTAs of the GEMM:
        // 18.8 us with 16 CTAs here, 19.2 with 128).
        const int room = sm_count() - n_tiles * m_tiles, most = n_tiles * m_tiles >= sm_count() ? INT32_MAX : room > 32 ? room : 32;
        int toks = 1;
        while (toks < 8 && (mpad / toks > most || g.nchunks * (KC / 4) * toks * 2 <= 4 * 256)) toks <<= 1;
        while (toks > 1 && (int64_t) g.nchunks * (KC / 4) * toks > (int64_t) PREP_MAX_V * 256) toks >>= 1;
        // Where many of them would meet on the SMs that the predecessor's last wave leaves free (behind one another such products are resident together),
        // eight tokens a CTA and so many registers that an SM takes one.  us, 32 float4 a thread always / with the lines above alone / now: Q4_0 2048 x 4048, 512 tokens
        // 18.9 / 21.6 / 18.8; 512 x 12288, 700 tokens 30.6 / 31.8 / 30.6; 2048 x 8192, 512 tokens 31.4 / 32.7 / 31.3.  Rows of 256 weights are over before that
        // matters (256 x 4048, 512 tokens 12.3 / 11.4).
        const int idle = sm_count() - 1 - (n_tiles * m_tiles - 1) % sm_count();
        const bool crowd = toks > 1 && mpad / toks > 3 * idle && g.nchunks * KC > 256;
        if (crowd)
            while (toks < 8 && g.nchunks * (KC / 4) * toks * 2 <= PREP_MAX_V * 256) toks <<= 1;
        const int per = crowd ? PREP_MAX_V : (g.nchunks * (KC / 4) * toks + 255) / 256;
        auto prep = per <= 4 ? gemm_prep_x<TN, 4> : per <= 8 ? gemm_prep_x<TN, 8> : per <= 16 ? gemm_prep_x<TN, 16> : gemm_prep_x<TN, PREP_MAX_V>;
        st = launch(prep, dim3((unsigned) (mpad / toks)), dim3(256), 0, s, x + c0 * ldx, ldx, (int) mm, (int) k, g.nchunks, toks,
                    dtype == DT_Q4_K ? 0 : dtype == DT_Q4_0 ? 2 : 1, tokscale, xh);
        if (st != ST_OK) return st;
        g.xh = xh;
        g.tokscale = tokscale;
        g.y = y + c0 * g.ldy;
        g.m = (int) mm;
        g.m_tiles = m_tiles;
        st = launch_gemm_dtype<TN, STAGES, SUB>(s, dtype, layout, g, n_tiles);
        if (st != ST_OK) return st;
    }
    return ST_OK;
}

}  // namespace

// Tensor-core MUL_MAT.  *handled = false (and ST_OK) when the shape or dtype is left to the caller's fallback.
int gemm_tc_mul_mat(cudaStream_t s, int dtype, int layout, const void * w, int64_t w_row_stride, int64_t k, int64_t n, const float * x,
                    int64_t ldx, int64_t m, float * y, int64_t ldy, bool * handled) {
    *handled = false;
    const bool packed = layout == LAYOUT_PACKED;
    if (!(dtype == DT_Q8_0 || dtype == DT_Q4_0 || dtype == DT_F16 || (dtype == DT_Q4_K && packed))) return ST_OK;
    if (k % 32 != 0 || (dtype == DT_Q4_K && k % 256 != 0)) return ST_OK;
    if (n > INT32_MAX - TM || k > INT32_MAX - 128 || m > INT32_MAX / 2) return ST_OK;
    if ((((uintptr_t) x) & 15) != 0 || ldx % 4 != 0) return ST_OK;
    if (packed && (((uintptr_t) w) & 31) != 0) return ST_OK;
    const int be = block_elems(dtype);
    if (w_row_stride == 0) w_row_stride = k / be * block_bytes(dtype);

    const int n_tiles = (int) ((n + TM - 1) / TM);
    GemmArgs g = {};
    const int fw = fault_word(FAULT_GEMM, &g.fault);
    if (fw != ST_OK) return fw;
    g.w.base = (const uint8_t *) w;
    g.w.planes = packed ? planes_for(dtype, n, k) : Planes{};
    g.w.row_stride = w_row_stride;
    g.w.blocks_per_row = k / be;
    g.w.n = (int) n;
    g.w.last_block = (int) (k / 32) - 1;
    g.n = (int) n;
    g.ldy = ldy;
    // Tile choice.  128 weight rows x 256 tokens per CTA once such tiles fill the SMs: a 128 x 128 tile takes more than half the time, because
    // the MMA warp's hand-over from stage to stage shows (446 cycles a chunk with one chunk a stage, MMAs 256; two chunks a stage:
    // Q4_0 5003 x 77 tokens 26.2 -> 23.3 us, 4096 x 512 30.8 -> 27.7 us).
    static const int forced_tn = [] { const char * e = getenv("SM100_GEMM_TN"); return e != nullptr ? atoi(e) : 0; }();
    int tn = (int64_t) n_tiles * ((m + 255) / 256) >= (int64_t) sm_count() ? 256 : 128;
    if (forced_tn == 128 || forced_tn == 256) tn = forced_tn;
    // more activation stages than these in flight slow the weight loads down by more than they hide
    const int st = tn == 256 ? gemm_passes<256, 6, 1>(s, dtype, layout, g, x, ldx, m, k, y) : gemm_passes<128, 6, 2>(s, dtype, layout, g, x, ldx, m, k, y);
    if (st != ST_OK) return st;
    *handled = true;
    return ST_OK;
}

}  // namespace sm100
