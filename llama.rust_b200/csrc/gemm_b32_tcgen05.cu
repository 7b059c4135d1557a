// Mat-muls of many activation rows against Q8_0, Q4_0 and MXFP4 weights (32-element blocks) on the fifth-generation tensor cores.
//
//   acc = fma(dot(block), d_w d_x, acc) over a row's 32-element blocks in ascending order
//
// is the chain of the reference's 8x8 gemm (crates/ggml/src/repack.rs:3380-3421, :1136-1184) and of its MXFP4 form; for Q4_0 and MXFP4
// the results are the CPU route's bits.  The reference's Q8_0 route keeps eight lane sums per block (crates/ggml/src/tinyblas.rs:64-74,
// vec_dot.rs:732-752), so here Q8_0 differs by the order of f32 sums and belongs to the fast numerics mode.
//
// Operands are f16: an activation, a Q8_0 weight, a nibble minus 8 and twice an E2M1 code are small integers, and a block's dot (at most 32 x
// 128 x 128) is an exact f32 sum, whatever the order.  tcgen05 kind::f16 leaves the dots in tensor memory as floats; kind::i8 would
// take half the tensor core's time (64 against 128 cycles per block of a 128 x 128 tile) but leave int32, whose conversion costs the drain a
// third instruction per element.
//
// Tiles of 128 weight rows x NC activation rows, walked by persistent CTAs, one per SM; a pipeline step is two blocks (K = 64).
//   warps 0 .. 7    drain: warp w owns weight rows 32 (w % 4) .. and columns NC / 2 (w / 4) ..; per block d_w d_x, then the fma, two columns
//                   per instruction
//   warp 8          one thread issues two K = 16 MMAs per block into one of TS tensor-memory stages of NC columns
//   warp 9          (one thread) copies the step's activations, 64 f16 of NC rows, by TMA, and their scales, which have slots and barriers of
//                   their own: the MMAs take the ones, the drain waits for the others
//   warps 12 .. 19  produce the weights' operand: a thread per row and block of the step
// The activations come as f16 from their quantizer (ActF16): rows of K values, the elements of each 8 in the order 0 2 1 3 4 6 5 7 in which the
// producers' unpacking yields them, in the block that holds the quantized rows: calls with blocks of their own share nothing.
//
// What bounds it: the handing over of blocks and shared memory.  A block of a 128 x 128 tile takes 900 cycles (Q8_0, 14336 x 4096 on 512 rows); its
// MMAs take 128, the drain's lanes 256 (a multiply and an fma per output; 53 % of the issue slots are used in all), shared memory about 610
// wavefronts: 290 of loads (activation scales, barriers) and 120 of stores (weights) as counted, 128 for the MMAs' operands and 70 for the
// copies as worked out.  The 128-column instances of Q8_0 and MXFP4 spill 40 and 28 bytes.  Tried and slower: 16 draining warps (far more
// spills at 128 columns; 64 columns 50 -> 53 us), the scales
// brought to tensor memory by an MMA with a row of ones (4096 x 4096 on 64 rows 50 -> 66 us, 14336 x 4096 on 512 263 -> 271).
// Every wait is bounded; a wait that runs out raises the CTA's abort flag and the device error word.
#include <cuda_fp16.h>

#include "common.cuh"
#include "tensor_map.h"

namespace b200 {

namespace {

constexpr int BQ_ROWS = 128, BQ_EPI_WARPS = 8, BQ_MMA_WARP = 8, BQ_LOAD_WARP = 9, BQ_PROD_WARP0 = 12, BQ_PROD_WARPS = 8;
constexpr int BQ_THREADS = (BQ_PROD_WARP0 + BQ_PROD_WARPS) * 32;   // launched with 96 registers a thread: 61440 for the CTA
constexpr int BQ_A_STEP = BQ_ROWS * 128;
constexpr uint32_t BQ_WAIT_LIMIT = 1u << 22;
constexpr int BQ_ERR_WAIT = 4;

template <int NC>
struct BqCfg {
    static constexpr int B_STEP = NC * 128, STAGE = BQ_A_STEP + B_STEP;
    static constexpr int STAGES = NC == 128 ? 6 : 8;
    static constexpr int TS = 256 / NC, TCOLS = 2 * NC;   // tensor-memory stages: the two blocks of a step next to each other
    // scale slots: when a stage comes free (its MMAs are done) the drain may still be in the step TS steps behind it
    static constexpr int DSLOTS = 16, DSLOT = 2 * NC * 4;
    static_assert(DSLOTS > STAGES + TS, "scale slots");
    static constexpr int SMEM = STAGES * STAGE + DSLOTS * DSLOT + 1024;   // 214016, 205824
    // two warpgroups drain, one holds the single-thread roles, two produce: the sum stays within the 5 x 96 registers of the launch
    static constexpr int REGS_EPI = NC == 128 ? 152 : 144, REGS_CTL = 40, REGS_PROD = NC == 128 ? 64 : 72;
    static_assert(2 * REGS_EPI + REGS_CTL + 2 * REGS_PROD <= 5 * 96, "register split");
    // kind::f16 instruction descriptor: f32 accumulator, f16 x f16, both operands K-major, N = NC, M = 128
    static constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NC >> 3) << 17) | ((uint32_t)(BQ_ROWS >> 4) << 24);
};
template <int NC>
struct alignas(16) BqBars {
    uint64_t afull[8], bfull[8], empty[8], tfull[4], tempty[4], dfull[BqCfg<NC>::DSLOTS];
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ uint32_t bq_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint64_t bq_desc(uint32_t addr) {   // K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
    return (uint64_t)((addr >> 4) & 0x3fffu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void bq_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bq_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bq_arrive(uint64_t *bar) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(bq_smem(bar)) : "memory");
}
__device__ __forceinline__ void bq_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bq_poll(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bq_smem(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool bq_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
    for (uint32_t it = 0; it < BQ_WAIT_LIMIT; it++) {
        if (bq_poll(bar, parity)) return true;
        if ((it & 255) == 255 && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void bq_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d_tmem), "l"(adesc), "l"(bdesc),
                 "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void bq_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bq_smem(bar)) : "memory");
}
// 32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void bq_ld32(uint32_t (&r)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ unsigned long long bq_bits(float2 v) { return *reinterpret_cast<unsigned long long *>(&v); }
__device__ __forceinline__ float2 bq_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(*reinterpret_cast<unsigned long long *>(&d)) : "l"(bq_bits(a)), "l"(bq_bits(b)), "l"(bq_bits(c)));
    return d;
}
__device__ __forceinline__ float2 bq_mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(*reinterpret_cast<unsigned long long *>(&d)) : "l"(bq_bits(a)), "l"(bq_bits(b)));
    return d;
}
__device__ __forceinline__ uint32_t bq_h2(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ __half2 bq_as_h2(uint32_t u) { return *reinterpret_cast<__half2 *>(&u); }
// signed bytes 0 and 2 (shift 0) or 1 and 3 (shift 8) of the word as f16: (1024 + (y ^ 0x80)) - 1152, exact
__device__ __forceinline__ uint32_t bq_signed(uint32_t y, int shift) {
    return bq_h2(__hsub2(bq_as_h2((((y ^ 0x80808080u) >> shift) & 0x00ff00ffu) | 0x64006400u), __float2half2_rn(1152.0f)));
}
// low (HI 0) or high nibbles of bytes 0 and 2 (ODD 0) or 1 and 3 as f16
template <int TYPE, int HI, int ODD>
__device__ __forceinline__ uint32_t bq_nibbles(uint32_t x) {
    if constexpr (TYPE == B200_TYPE_Q4_0) {
        const uint32_t y = ODD ? x >> 8 : x;
        if constexpr (HI) return bq_h2(__hfma2(bq_as_h2((y & 0x00f000f0u) | 0x64006400u), __float2half2_rn(0.0625f), __float2half2_rn(-72.0f)));   // (1024 + 16 w) / 16 - 72
        return bq_h2(__hsub2(bq_as_h2((y & 0x000f000fu) | 0x64006400u), __float2half2_rn(1032.0f)));
    } else {
        // E2M1 code s e e m: sign, two exponent bits and the mantissa bit in an f16's places make 2^-15 of twice its value (zero and one half
        // as subnormals)
        constexpr int at = 8 * ODD + 4 * HI, up = 9 - at, sg = 12 - at;
        const uint32_t em = (up >= 0 ? x << (up & 31) : x >> (-up & 31)) & 0x0e000e00u, s = (x << sg) & 0x80008000u;
        return bq_h2(__hmul2(bq_as_h2(em | s), __float2half2_rn(32768.0f)));
    }
}

template <int TYPE, int NC>
__global__ void __launch_bounds__(BQ_THREADS, 1)
gemm_b32_tcgen05_kernel(const __grid_constant__ CUtensorMap xmap, const uint8_t *__restrict__ tiles, const float *__restrict__ scales, int64_t ld_scale, float *dst,
                        int64_t lddst, int64_t n, int nb, int64_t m, int row_blocks, int col_blocks, int *err) {
    using C = BqCfg<NC>;
    constexpr int S = C::STAGES, TS = C::TS, CPT = NC / 2;
    constexpr int CHUNK = TYPE == B200_TYPE_Q8_0 ? 8704 : TYPE == B200_TYPE_Q4_0 ? 4608 : 4352;   // bytes of a 32-row tile's 256-element group
    constexpr int SC_OFF = TYPE == B200_TYPE_Q8_0 ? 8192 : 4096;
    extern __shared__ uint8_t bq_raw[];
    __shared__ BqBars<NC> bars;
    pdl_trigger();
    const uint32_t smem = (bq_smem(bq_raw) + 1023u) & ~1023u;
    uint8_t *const smem_p = bq_raw + (smem - bq_smem(bq_raw));
    float *const da = reinterpret_cast<float *>(smem_p + S * C::STAGE);   // [DSLOTS][2][NC]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    volatile int *abort_flag = &bars.abort_flag;
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; i++) {
            bq_init(&bars.afull[i], BQ_PROD_WARPS / 2);
            bq_init(&bars.bfull[i], 1);
            bq_init(&bars.empty[i], 1);
        }
        for (int i = 0; i < TS; i++) {
            bq_init(&bars.tfull[i], 1);
            bq_init(&bars.tempty[i], BQ_EPI_WARPS);
        }
        for (int i = 0; i < C::DSLOTS; i++) bq_init(&bars.dfull[i], 1);
        bars.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == BQ_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bq_smem(&bars.tmem_base)), "r"(TS * C::TCOLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = bars.tmem_base;
    const int total = row_blocks * col_blocks;   // the column blocks of a row block are adjacent
    const int64_t tiles_n = (n + TILE_ROWS - 1) / TILE_ROWS;
    const int ksteps = 4 * nb;

    if (warp < BQ_EPI_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::REGS_EPI));
        pdl_wait();   // the previous kernels in the stream may still read dst
        const int q = warp & 3, h = warp >> 2;
        const uint32_t trow0 = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(CPT * h);
        constexpr int SCB = TYPE == B200_TYPE_MXFP4 ? 2 : 4;   // bytes of a row's two scales of a step
        float2 acc[CPT / 2];
        int step = 0;   // steps done by this CTA
        bool ok = true;
        // step p's dots are in tensor memory, and its activation scales in their slot: a copy of their own, of which the dots being there says
        // nothing.  The slot is not filled again before this warp has left the step, so its phase cannot run ahead
        const auto ready = [&](int p) {
            const bool r = __all_sync(0xffffffffu, bq_wait(&bars.tfull[p % TS], (uint32_t)(p / TS) & 1u, abort_flag) &&
                                                       bq_wait(&bars.dfull[p % C::DSLOTS], (uint32_t)(p / C::DSLOTS) & 1u, abort_flag));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return r;
        };
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            const int rb = t / col_blocks, cb = t - rb * col_blocks;
            const int64_t tile = (int64_t)rb * (BQ_ROWS / TILE_ROWS) + q;
            const bool row_ok = tile < tiles_n;
            const uint8_t *sc = tiles + (row_ok ? tile : 0) * (int64_t)nb * CHUNK + SC_OFF + lane * 4 * SCB;
            const auto load_scales = [&](int ks) -> uint32_t {
                const uint8_t *p = sc + (int64_t)(ks >> 2) * CHUNK + (ks & 3) * SCB;
                return !row_ok ? 0u : TYPE == B200_TYPE_MXFP4 ? (uint32_t) * (const uint16_t *)p : *(const uint32_t *)p;
            };
            uint32_t ws_next = load_scales(0);
#pragma unroll
            for (int c = 0; c < CPT / 2; c++) acc[c] = make_float2(0.0f, 0.0f);
            // rounds of 32 columns of one block, RN a step; the next round's are on their way while one is added: v[round % 2]
            constexpr int RN = 2 * CPT / 32;
            uint32_t v[2][32];
            if (!(ok = ready(step))) break;
            bq_ld32(v[0], trow0 + (uint32_t)((step % TS) * C::TCOLS));
            for (int ks = 0; ks < ksteps; ks++, step++) {
                const uint32_t ws = ws_next;
                if (ks + 1 < ksteps) ws_next = load_scales(ks + 1);
                const float4 *das = reinterpret_cast<const float4 *>(da + (size_t)(step % C::DSLOTS) * 2 * NC + CPT * h);
                const uint32_t trow = trow0 + (uint32_t)((step % TS) * C::TCOLS);
#pragma unroll
                for (int r = 0; r < RN; r++) {
                    const int blk = r / (RN / 2), col = (r % (RN / 2)) * 32;
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    bool early = true;
                    if (r + 1 < RN) {
                        bq_ld32(v[(r + 1) & 1], trow + (uint32_t)((r + 1) / (RN / 2) * NC + (r + 1) % (RN / 2) * 32));
                    } else {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) bq_arrive(&bars.tempty[step % TS]);
                        // the next step's first round, if its dots (and scales) are there already
                        early = ks + 1 == ksteps;
                        if (!early) {
                            const bool dots = bq_poll(&bars.tfull[(step + 1) % TS], (uint32_t)((step + 1) / TS) & 1u);
                            const bool scales_in = bq_poll(&bars.dfull[(step + 1) % C::DSLOTS], (uint32_t)((step + 1) / C::DSLOTS) & 1u);
                            early = __all_sync(0xffffffffu, dots && scales_in);
                        }
                        if (early && ks + 1 < ksteps) {
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            bq_ld32(v[0], trow0 + (uint32_t)(((step + 1) % TS) * C::TCOLS));
                        }
                    }
                    const float dw = TYPE == B200_TYPE_MXFP4 ? e8m0_half_to_f32((ws >> (8 * blk)) & 0xffu) : f16_bits_to_f32((uint16_t)(blk ? ws >> 16 : ws & 0xffffu));
                    const float2 dw2 = make_float2(dw, dw);
#pragma unroll
                    for (int c4 = 0; c4 < 8; c4++) {
                        const float4 dq = das[(blk * NC + col) / 4 + c4];
                        const float2 s0 = bq_mul2(make_float2(dq.x, dq.y), dw2), s1 = bq_mul2(make_float2(dq.z, dq.w), dw2);
                        float2 *a = acc + col / 2 + 2 * c4;
                        a[0] = bq_fma2(make_float2(__uint_as_float(v[r & 1][4 * c4]), __uint_as_float(v[r & 1][4 * c4 + 1])), s0, a[0]);
                        a[1] = bq_fma2(make_float2(__uint_as_float(v[r & 1][4 * c4 + 2]), __uint_as_float(v[r & 1][4 * c4 + 3])), s1, a[1]);
                    }
                    if (!early) {
                        if (!(ok = ready(step + 1))) break;
                        bq_ld32(v[0], trow0 + (uint32_t)(((step + 1) % TS) * C::TCOLS));
                    }
                }
                if (!ok) break;
            }
            const int64_t row = tile * TILE_ROWS + lane;
            if (!ok || !row_ok || row >= n) continue;
#pragma unroll
            for (int c = 0; c < CPT; c++) {
                const float v = (c & 1) ? acc[c >> 1].y : acc[c >> 1].x;
                const int64_t col = (int64_t)cb * NC + CPT * h + c;
                if (col < m) dst[col * lddst + row] = v;
            }
        }
    } else if (warp >= BQ_PROD_WARP0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::REGS_PROD));
        const int pw = warp - BQ_PROD_WARP0, odd = pw >> 2, tt = pw & 3, prow = tt * 32 + lane, sw = prow & 7;
        uint8_t *const a0 = smem_p + prow * 128;
        constexpr int PIECES = TYPE == B200_TYPE_Q8_0 ? 4 : 2;   // 16-byte pieces of a step's two blocks
        // the chunk of 256-element group b of tile t (its row tile tt), nullptr past the work's end or the matrix's last row tile
        const auto chunk_of = [&](int t, int b) -> const uint8_t * {
            if (t >= total) return nullptr;
            const int64_t tile = (int64_t)(t / col_blocks) * (BQ_ROWS / TILE_ROWS) + tt;
            if (tile >= tiles_n) return nullptr;
            return tiles + (tile * nb + b) * (int64_t)CHUNK;
        };
        const auto next = [&](int &t, int &b) {
            if (++b == nb) {
                b = 0;
                t += gridDim.x;
            }
        };
        uint4 w[2][PIECES];
        const auto fetch = [&](const uint8_t *c, int g) {   // this warp's g-th step of the group
#pragma unroll
            for (int i = 0; i < PIECES; i++)
                w[g][i] = c ? ld_stream16(c + ((2 * g + odd) * PIECES + i) * 512 + lane * 16) : make_uint4(0, 0, 0, 0);
        };
        const auto ahead = [&](const uint8_t *c) {   // the two warps of a row tile ask L2 for its chunk
            if (c)
                for (int l = lane + 32 * odd; l * 128 < CHUNK; l += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(c + l * 128));
        };
        int t = blockIdx.x, b = 0, t1 = t, b1 = 0, ta = t, ba = 0;   // this group, the next one, and one that L2 is asked for
        for (int i = 0; i < 3; i++) {
            ahead(chunk_of(ta, ba));
            next(ta, ba);
        }
        const uint8_t *cur = chunk_of(t, b);
        fetch(cur, 0);
        fetch(cur, 1);
        int step = odd;
        bool ok = true;
        while (t < total && ok) {
            next(t1, b1);
            const uint8_t *nxt = chunk_of(t1, b1);
            ahead(chunk_of(ta, ba));
            next(ta, ba);
#pragma unroll
            for (int g = 0; g < 2; g++, step += 2) {
                const int s = step % S;
                if (!__all_sync(0xffffffffu, bq_wait(&bars.empty[s], ((uint32_t)(step / S) & 1u) ^ 1u, abort_flag))) {
                    ok = false;
                    break;
                }
                uint8_t *dstp = a0 + s * C::STAGE;
                const auto put = [&](int c, uint32_t u0, uint32_t u1, uint32_t u2, uint32_t u3) {
                    *reinterpret_cast<uint4 *>(dstp + ((c ^ sw) << 4)) = make_uint4(u0, u1, u2, u3);
                };
#pragma unroll
                for (int i = 0; i < PIECES; i++) {
                    const uint4 p = w[g][i];
                    if constexpr (TYPE == B200_TYPE_Q8_0) {
                        put(2 * i, bq_signed(p.x, 0), bq_signed(p.x, 8), bq_signed(p.y, 0), bq_signed(p.y, 8));
                        put(2 * i + 1, bq_signed(p.z, 0), bq_signed(p.z, 8), bq_signed(p.w, 0), bq_signed(p.w, 8));
                    } else {
                        put(4 * i, bq_nibbles<TYPE, 0, 0>(p.x), bq_nibbles<TYPE, 0, 1>(p.x), bq_nibbles<TYPE, 0, 0>(p.y), bq_nibbles<TYPE, 0, 1>(p.y));
                        put(4 * i + 1, bq_nibbles<TYPE, 0, 0>(p.z), bq_nibbles<TYPE, 0, 1>(p.z), bq_nibbles<TYPE, 0, 0>(p.w), bq_nibbles<TYPE, 0, 1>(p.w));
                        put(4 * i + 2, bq_nibbles<TYPE, 1, 0>(p.x), bq_nibbles<TYPE, 1, 1>(p.x), bq_nibbles<TYPE, 1, 0>(p.y), bq_nibbles<TYPE, 1, 1>(p.y));
                        put(4 * i + 3, bq_nibbles<TYPE, 1, 0>(p.z), bq_nibbles<TYPE, 1, 1>(p.z), bq_nibbles<TYPE, 1, 0>(p.w), bq_nibbles<TYPE, 1, 1>(p.w));
                    }
                }
                fetch(nxt, g);
                // the stores (generic proxy) before the tensor core's reads (async proxy), then the warp's arrival
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) bq_arrive(&bars.afull[s]);
            }
            t = t1;
            b = b1;
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::REGS_CTL));
        if (warp == BQ_MMA_WARP) {
            if (lane == 0) {
                int step = 0;
                bool ok = true;
                for (int t = blockIdx.x; t < total && ok; t += gridDim.x)
                    for (int ks = 0; ks < ksteps; ks++, step++) {
                        const int s = step % S, ts = step % TS;
                        const uint32_t ph = (uint32_t)(step / S) & 1u;
                        if (!bq_wait(&bars.tempty[ts], ((uint32_t)(step / TS) & 1u) ^ 1u, abort_flag) || !bq_wait(&bars.bfull[s], ph, abort_flag) ||
                            !bq_wait(&bars.afull[s], ph, abort_flag)) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t stage = smem + (uint32_t)(s * C::STAGE);
                        const uint64_t ad = bq_desc(stage), bd = bq_desc(stage + BQ_A_STEP);
#pragma unroll
                        for (int i = 0; i < 4; i++)   // K = 16 step i: 32 bytes on; two make a block
                            bq_mma(tmem + (uint32_t)(ts * C::TCOLS + (i >> 1) * NC), ad + 2 * i, bd + 2 * i, C::IDESC, i & 1);
                        bq_commit(&bars.tfull[ts]);
                        bq_commit(&bars.empty[s]);
                    }
            }
        } else if (warp == BQ_LOAD_WARP && lane == 0) {
            pdl_wait();   // the activations are the previous kernel's output
            int step = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
                const int cb = t % col_blocks;
                for (int ks = 0; ks < ksteps; ks++, step++) {
                    const int s = step % S;
                    if (!bq_wait(&bars.empty[s], ((uint32_t)(step / S) & 1u) ^ 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = bq_smem(&bars.bfull[s]), ds = bq_smem(da + (size_t)(step % C::DSLOTS) * 2 * NC), dbar = bq_smem(&bars.dfull[step % C::DSLOTS]);
                    bq_expect(bar, C::B_STEP);
                    bq_expect(dbar, C::DSLOT);
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                                     smem + (uint32_t)(s * C::STAGE + BQ_A_STEP)),
                                 "l"(&xmap), "r"(ks * 64), "r"(cb * NC), "r"(bar)
                                 : "memory");
#pragma unroll
                    for (int i = 0; i < 2; i++)
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(ds + (uint32_t)(i * NC * 4)),
                                     "l"(scales + (int64_t)(2 * ks + i) * ld_scale + (int64_t)cb * NC), "r"(NC * 4), "r"(dbar)
                                     : "memory");
                }
            }
            // the copies in flight, also when this CTA gave up
            for (int p = step < S ? 0 : step - S; p < step; p++)
                for (uint32_t it = 0; it < BQ_WAIT_LIMIT; it++)
                    if (bq_poll(&bars.bfull[p % S], (uint32_t)(p / S) & 1u) && bq_poll(&bars.dfull[p % C::DSLOTS], (uint32_t)(p / C::DSLOTS) & 1u)) break;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == BQ_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TS * C::TCOLS) : "memory");
    }
    if (threadIdx.x == 0 && bars.abort_flag) atomicExch(err, BQ_ERR_WAIT);
}

struct BqCall {
    int64_t n, k, m;
    const uint8_t *tiles;
    float *dst;
    int64_t lddst;
    ActF16 acts;
    int64_t row_blocks, col_blocks;
};

template <int TYPE, int NC>
int launch_b32(const BqCall &c, int sms, cudaStream_t s) {
    static bool attr_done[64] = {false};
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    B200_REQUIRE(dev >= 0 && dev < 64, "gemm: device index %d out of range", dev);
    if (!attr_done[dev]) {
        B200_CUDA(cudaFuncSetAttribute(gemm_b32_tcgen05_kernel<TYPE, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, BqCfg<NC>::SMEM));
        attr_done[dev] = true;
    }
    int *err = nullptr;
    int rc = device_error_word(&err);
    if (rc != B200_STATUS_SUCCESS) return rc;
    CUtensorMap xmap;
    rc = rows_map(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, c.acts.x, c.k, c.m, c.k, NC);
    if (rc != B200_STATUS_SUCCESS) return rc;
    const int64_t tiles = c.row_blocks * c.col_blocks;
    return launch_pdl(gemm_b32_tcgen05_kernel<TYPE, NC>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(BQ_THREADS), (size_t)BqCfg<NC>::SMEM, s, xmap, c.tiles, (const float *)c.acts.scales,
                      c.acts.ld, c.dst, c.lddst, c.n, (int)(c.k / GROUP_K), c.m, (int)c.row_blocks, (int)c.col_blocks, err);
}
template <int TYPE>
int launch_b32_nc(int nc, const BqCall &c, int sms, cudaStream_t s) {
    return nc == 128 ? launch_b32<TYPE, 128>(c, sms, s) : launch_b32<TYPE, 64>(c, sms, s);
}

// ns of a wave of tiles per 32-element block, with 64 and 128 columns (4096 x 4096 on 256 rows 48 us, on 512 rows 72 us), and of the int8
// kernel's 32 columns (4096 x 4096 on 64 rows 31 us; MXFP4 38)
constexpr int BQ_WAVE_64 = 350, BQ_WAVE_128 = 500, BQ_WAVE_I8 = 200, BQ_WAVE_I8_MXFP4 = 260;
int64_t b32_waves(int64_t row_blocks, int64_t m, int nc, int sms) { return (row_blocks * ((m + nc - 1) / nc) + sms - 1) / sms; }
int b32_columns(int64_t row_blocks, int64_t m, int sms) {
    return b32_waves(row_blocks, m, 128, sms) * BQ_WAVE_128 < b32_waves(row_blocks, m, 64, sms) * BQ_WAVE_64 ? 128 : 64;
}

}  // namespace

int sm_count() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    return sms;
}

// the columns of launch_gemm_b32's tiles where it is the quicker one, else 0: the int8 kernel (gemm_tcgen05_i8.cu) has tiles of 32 columns, which
// pays while they make few waves.  Same results.  us of a call with the int8 kernel and with this one, Q8_0: 14336 x 4096 on 512 rows
// 367, 262 (MXFP4 442, 239); 8816 x 2304 on 107 37, 33; 2488 x 1024 on 307 22, 18; and the other way 4096 x 4096 on 128 32, 50; 23288 x 11520 on
// 134 466, 487
int gemm_b32_pick_for(int type, int64_t n, int64_t m, int sms) {
    const int64_t row_blocks = (n + BQ_ROWS - 1) / BQ_ROWS;
    const int nc = b32_columns(row_blocks, m, sms);
    const int64_t here = b32_waves(row_blocks, m, nc, sms) * (nc == 128 ? BQ_WAVE_128 : BQ_WAVE_64);
    return here < b32_waves(row_blocks, m, 32, sms) * (type == B200_TYPE_MXFP4 ? BQ_WAVE_I8_MXFP4 : BQ_WAVE_I8) ? nc : 0;
}
bool gemm_b32_wins(int type, int64_t n, int64_t m) { return gemm_b32_pick_for(type, n, m, sm_count()) != 0; }

// Q8_0 (fast numerics), Q4_0 and MXFP4 (8x8 gemm chain) mat-muls
int launch_gemm_b32(int type, int64_t n, int64_t k, int64_t m, const uint8_t *tiles, ActF16 acts, float *dst, int64_t lddst, cudaStream_t s) {
    B200_REQUIRE(k % GROUP_K == 0, "gemm: k = %lld must be a multiple of 256", (long long)k);
    if (n == 0 || m == 0) return B200_STATUS_SUCCESS;
    const int64_t row_blocks = (n + BQ_ROWS - 1) / BQ_ROWS;
    const int sms = sm_count(), nc = b32_columns(row_blocks, m, sms);
    BqCall c = {};
    c.n = n; c.k = k; c.m = m; c.tiles = tiles; c.dst = dst; c.lddst = lddst; c.acts = acts;
    c.row_blocks = row_blocks;
    c.col_blocks = (m + nc - 1) / nc;
    B200_REQUIRE(c.row_blocks * c.col_blocks < (1ll << 31) - (1 << 20), "gemm: %lld x %lld is too large for one launch", (long long)n, (long long)m);
    B200_REQUIRE(acts.x && acts.ld >= c.col_blocks * nc, "gemm: no f16 activations for %lld rows", (long long)m);
    switch (type) {
        case B200_TYPE_Q8_0: return launch_b32_nc<B200_TYPE_Q8_0>(nc, c, sms, s);
        case B200_TYPE_Q4_0: return launch_b32_nc<B200_TYPE_Q4_0>(nc, c, sms, s);
        case B200_TYPE_MXFP4: return launch_b32_nc<B200_TYPE_MXFP4>(nc, c, sms, s);
        default: B200_REQUIRE(false, "gemm: weight type %d has no 32-element blocks", type);
    }
}

}  // namespace b200
