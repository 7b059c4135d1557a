// BF16 x BF16 mat-mul on the tensor cores for many activation rows: y[m][n] = act(w[n][k] x[m][k] + bias) + addend, F32 sums.
//
// Output tiles of 128 weight rows x NC activation rows (64, 128 or 256), or of 256 x 256 by pairs of CTAs (further down), walked by persistent
// CTAs, one per SM, the column blocks of a weight row block next to each other so that the weights cross HBM once.  Per tile a pipeline of K = 64 steps: one thread moves the
// two operand boxes with TMA (128-byte swizzle; the hardware fills what lies outside either matrix with zeros), one thread issues four
// M 128 x N NC x K 16 MMAs per step into one of two tensor-memory stages, four warps drain the other stage: lane = weight row, so a
// store of one activation row's 32 outputs is one contiguous piece.  The activation function and the residual add are done there;
// a gated one takes neighbouring weight rows (gate, up), which neighbouring lanes exchange, each keeping every other activation row.
// Every wait is bounded; a wait that runs out raises the CTA's abort flag and the device error word.
#include "dense.cuh"
#include "tensor_map.h"

namespace b200 {

typedef CUresult (*encode_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                              const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static encode_fn tensor_map_encoder() {
    static encode_fn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (encode_fn)p;
        else cudaGetLastError();
    }
    return fn;
}
int rows_map(CUtensorMap *map, CUtensorMapDataType type, const void *base, int64_t k, int64_t rows, int64_t ld, int box_rows) {
    encode_fn enc = tensor_map_encoder();
    B200_REQUIRE(enc != nullptr, "gemm: the driver has no tensor-map encoder");
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, es[2] = {1, 1};
    const CUresult r = enc(map, type, 2, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200_REQUIRE(r == CUDA_SUCCESS, "gemm: tensor map of %lld x %lld (stride %lld) refused (%d)", (long long)rows, (long long)k, (long long)ld, (int)r);
    return B200_STATUS_SUCCESS;
}
bool cache_tile_map(CUtensorMap *map, const void *base, int64_t d, int64_t heads, int64_t n_pos, int64_t nb1, int64_t nb2, int box_pos) {
    encode_fn enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)n_pos}, strides[2] = {(cuuint64_t)nb2, (cuuint64_t)nb1};
    const cuuint32_t box[3] = {64, 1, (cuuint32_t)box_pos}, es[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

namespace {

constexpr int GB_ROWS = 128, GB_K = 64, GB_THREADS = 256, GB_EPI_WARP0 = 4, GB_TSTAGES = 2;
constexpr uint32_t GB_WAIT_LIMIT = 1u << 22;
constexpr int GB_ERR_WAIT = 4;

template <int NC>
struct GbCfg {
    static constexpr int A_BYTES = GB_ROWS * GB_K * 2, B_BYTES = NC * GB_K * 2, STAGE = A_BYTES + B_BYTES;
    static constexpr int STAGES = NC == 256 ? 4 : NC == 128 ? 6 : 8;
    static constexpr int SMEM = STAGES * STAGE + 1024;
    // kind::f16 instruction descriptor: F32 accumulator, BF16 x BF16, both operands K-major, N = NC, M = 128
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NC >> 3) << 17) | ((uint32_t)(GB_ROWS >> 4) << 24);
};
struct GbBars {
    uint64_t full[8], empty[8], tfull[GB_TSTAGES], tempty[GB_TSTAGES];
    uint32_t tmem_base;
    int abort_flag;
};
struct GbOut {
    void *y;
    int y_type;
    int64_t ldy;
    const float *addend;
    int64_t ld_addend;
    const float *bias;
    int act;
    float act_limit, act_alpha;
    int n, m;
};

__device__ __forceinline__ uint32_t gb_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint64_t gb_desc(uint32_t addr) {   // K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
    return (uint64_t)((addr >> 4) & 0x3fffu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void gb_bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void gb_bar_arrive(uint32_t bar) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gb_bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool gb_bar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    for (uint32_t it = 0; it < GB_WAIT_LIMIT; it++) {
        uint32_t ok;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((it & 255) == 255 && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void gb_tma_load(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x),
                 "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void gb_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d_tmem), "l"(adesc), "l"(bdesc),
                 "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void gb_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gb_tmem_ld32(uint32_t (&r)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// columns [c_begin, c_end) (multiples of 32) of this thread's tensor-memory lane: weight row `row` against activation rows col0 + c.
// read() is called by the whole warp once all of them are in registers
template <typename Read>
__device__ __forceinline__ void gb_drain(const GbOut &o, uint32_t trow, int row, int col0, int c_begin, int c_end, Read read) {
    const int lane = threadIdx.x & 31;
    const bool row_ok = row < o.n;
    const float bias = o.bias && row_ok ? o.bias[row] : 0.0f;
#pragma unroll 1
    for (int c0 = c_begin; c0 < c_end; c0 += 32) {
        uint32_t v[32];
        float ad[32];
        gb_tmem_ld32(v, trow + (uint32_t)c0);
        if (o.addend) {
#pragma unroll
            for (int c = 0; c < 32; c++) {
                const int col = col0 + c0 + c;
                ad[c] = row_ok && col < o.m ? o.addend[(int64_t)col * o.ld_addend + row] : 0.0f;
            }
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 >= c_end) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            read();
        }
        if (o.act == ACT_CLAMPED_GATE) {
            const int odd = lane & 1;
#pragma unroll
            for (int c = 0; c < 32; c += 2) {
                const float x0 = __uint_as_float(v[c]) + bias, x1 = __uint_as_float(v[c + 1]) + bias;
                const float other = __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 1);
                const float r = clamped_gate(odd ? other : x0, odd ? x1 : other, o.act_limit, o.act_alpha);
                const int col = col0 + c0 + c + odd;
                if (!row_ok || col >= o.m) continue;
                if (o.y_type == B200_TYPE_F32) ((float *)o.y)[(int64_t)col * o.ldy + (row >> 1)] = r;
                else ((__nv_bfloat16 *)o.y)[(int64_t)col * o.ldy + (row >> 1)] = __float2bfloat16_rn(r);
            }
            continue;
        }
        if (!row_ok) continue;
#pragma unroll
        for (int c = 0; c < 32; c++) {
            const int col = col0 + c0 + c;
            if (col >= o.m) break;
            float r = dense_act(o.act, __uint_as_float(v[c]) + bias);
            if (o.addend) r += ad[c];
            if (o.y_type == B200_TYPE_F32) ((float *)o.y)[(int64_t)col * o.ldy + row] = r;
            else ((__nv_bfloat16 *)o.y)[(int64_t)col * o.ldy + row] = __float2bfloat16_rn(r);
        }
    }
}

template <int NC>
__global__ void __launch_bounds__(GB_THREADS, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, GbOut o, int ksteps, int col_blocks, int tiles, int *err) {
    using C = GbCfg<NC>;
    constexpr int S = C::STAGES;
    extern __shared__ uint8_t gb_raw[];
    __shared__ GbBars bars;
    pdl_trigger();
    const uint32_t smem = (gb_smem(gb_raw) + 1023u) & ~1023u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    volatile int *abort_flag = &bars.abort_flag;
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; i++) {
            gb_bar_init(gb_smem(&bars.full[i]), 1);
            gb_bar_init(gb_smem(&bars.empty[i]), 1);
        }
        for (int i = 0; i < GB_TSTAGES; i++) {
            gb_bar_init(gb_smem(&bars.tfull[i]), 1);
            gb_bar_init(gb_smem(&bars.tempty[i]), 4);
        }
        bars.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        // both accumulator stages; the operand stages fill the SM's shared memory, so no second CTA competes for the columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gb_smem(&bars.tmem_base)), "r"(GB_TSTAGES * NC) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = bars.tmem_base;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            int step = 0, issued = -1;
            for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
                const int rb = t / col_blocks, cb = t - rb * col_blocks;
                bool ok = true;
                for (int ks = 0; ks < ksteps; ks++, step++) {
                    const int s = step % S;
                    if (!gb_bar_wait(gb_smem(&bars.empty[s]), ((uint32_t)(step / S) & 1u) ^ 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = gb_smem(&bars.full[s]), stage = smem + (uint32_t)(s * C::STAGE);
                    gb_bar_expect(bar, C::STAGE);
                    gb_tma_load(stage, &wmap, ks * GB_K, rb * GB_ROWS, bar);
                    gb_tma_load(stage + C::A_BYTES, &xmap, ks * GB_K, cb * NC, bar);
                    issued = step;
                }
                if (!ok) break;
            }
            // a CTA that gives up still waits (bounded) for the copies it has in flight
            if (*abort_flag)
                for (int p = issued - S + 1 < 0 ? 0 : issued - S + 1; p <= issued; p++) {
                    for (uint32_t it = 0; it < GB_WAIT_LIMIT; it++) {
                        uint32_t ok;
                        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                                     : "=r"(ok) : "r"(gb_smem(&bars.full[p % S])), "r"((uint32_t)(p / S) & 1u) : "memory");
                        if (ok) break;
                    }
                }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int step = 0, j = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, j++) {
                const int ts = j % GB_TSTAGES;
                if (!gb_bar_wait(gb_smem(&bars.tempty[ts]), ((uint32_t)(j / GB_TSTAGES) & 1u) ^ 1u, abort_flag)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_acc = tmem + (uint32_t)(ts * NC);
                for (int ks = 0; ks < ksteps; ks++, step++) {
                    const int s = step % S;
                    if (!gb_bar_wait(gb_smem(&bars.full[s]), (uint32_t)(step / S) & 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t stage = smem + (uint32_t)(s * C::STAGE);
                    const uint64_t ad = gb_desc(stage), bd = gb_desc(stage + C::A_BYTES);
#pragma unroll
                    for (int i = 0; i < GB_K / 16; i++) gb_mma(d_acc, ad + 2 * i, bd + 2 * i, C::IDESC, (ks | i) != 0);   // 32 bytes on per K = 16
                    gb_commit(gb_smem(&bars.empty[s]));
                }
                if (ok) gb_commit(gb_smem(&bars.tfull[ts]));
            }
        }
    } else if (warp >= GB_EPI_WARP0) {
        const int q = warp - GB_EPI_WARP0;   // tensor-memory lanes 32 q ..
        int j = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, j++) {
            const int rb = t / col_blocks, cb = t - rb * col_blocks, ts = j % GB_TSTAGES;
            if (!__all_sync(0xffffffffu, gb_bar_wait(gb_smem(&bars.tfull[ts]), (uint32_t)(j / GB_TSTAGES) & 1u, abort_flag))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = rb * GB_ROWS + 32 * q + lane, col0 = cb * NC;
            const uint32_t trow = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(ts * NC);
            gb_drain(o, trow, row, col0, 0, NC, [&] {
                if (lane == 0) gb_bar_arrive(gb_smem(&bars.tempty[ts]));
            });
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GB_TSTAGES * NC) : "memory");
    }
    if (threadIdx.x == 0 && bars.abort_flag) atomicExch(err, GB_ERR_WAIT);
}

// ---- pairs of SMs: more than 128 activation rows -----------------------------------------------------------------------------------------
// A tile of 256 weight rows x 256 activation rows is computed by the two CTAs of a cluster with one MMA per K = 16 (cta_group::2, M 256,
// N 256): each holds 128 of the weight rows and half of the activation rows in its shared memory and the sums of its weight rows in its
// tensor memory.  The even CTA's MMA thread issues for both.  Its `full` barrier counts the bytes of both CTAs' copies, its `tempty`
// barrier the epilogue warps of both; commits are multicast to both CTAs' `empty` and `tfull` barriers.
// What bounds it: the tensor cores (86 % of the active cycles on 14336 x 4096 x 2048 rows) at the clock that power leaves them (1.56 of
// 1.965 GHz there).  Why pairs: per K = 16 an SM's tensor core takes 128 cycles; a CTA alone on its 128 x 256 tile reads
// 12 KB and copies 12 KB in for it, 192 cycles at 128 bytes a cycle; a pair reads and copies 8 KB each, 128 cycles.  Against
// 128 x 256 tiles of single CTAs (us, a mat-mul alone): 8192 x 2048 x 2048 rows 62.0 -> 55.6, 14336 x 4096 x 2048 188.9 -> 170.5
// (1.41 PFLOP/s), 22016 x 4096 x 2048 278 -> 256.  Narrower pair tiles (N 224, 192, 160, 128) took longer from 1024 x 4096 x 2048 rows
// up.  Two epilogue warps share a quarter of the lanes: with K = 1024 one alone would take longer than the tile's MMAs.
constexpr int GP_EPI_WARPS = 8, GP_THREADS = 128 + GP_EPI_WARPS * 32, GP_STAGES = 6;
constexpr int GP_A_BYTES = GB_ROWS * GB_K * 2, GP_STAGE = 2 * GP_A_BYTES, GP_SMEM = GP_STAGES * GP_STAGE + 1024;
constexpr int GP_NC = 256;   // activation rows of a tile, tensor-memory columns of an accumulator stage
constexpr int GP_HALF = GP_NC / 2;
// kind::f16 instruction descriptor: F32 accumulator, BF16 x BF16, both operands K-major, N = 256, M = 256
constexpr uint32_t GP_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GP_NC >> 3) << 17) | ((uint32_t)(2 * GB_ROWS >> 4) << 24);

__device__ __forceinline__ uint32_t gp_of_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void gp_tma_load(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {   // bar: the leader's, a cluster address
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map),
                 "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int accumulate) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d_tmem), "l"(adesc), "l"(bdesc),
                 "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void gp_commit(uint32_t bar) {   // on this barrier of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void gp_arrive(uint32_t bar) {   // a cluster address
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(GP_THREADS, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, GbOut o, int ksteps, int col_blocks, int tiles, int *err) {
    constexpr int S = GP_STAGES;
    extern __shared__ uint8_t gb_raw[];
    __shared__ GbBars bars;
    pdl_trigger();
    const uint32_t smem = (gb_smem(gb_raw) + 1023u) & ~1023u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = (int)(blockIdx.x & 1), pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);   // clusters of two along x
    volatile int *abort_flag = &bars.abort_flag;
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; i++) {
            gb_bar_init(gb_smem(&bars.full[i]), 1);
            gb_bar_init(gb_smem(&bars.empty[i]), 1);
        }
        for (int i = 0; i < GB_TSTAGES; i++) {
            gb_bar_init(gb_smem(&bars.tfull[i]), 1);
            gb_bar_init(gb_smem(&bars.tempty[i]), 2 * GP_EPI_WARPS);
        }
        bars.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        // all columns of both SMs: the operand stages fill their shared memory, so no other CTA is waiting for some
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gb_smem(&bars.tmem_base)), "r"(GB_TSTAGES * GP_NC) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gp_cluster_sync();   // both CTAs' barriers stand
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = bars.tmem_base;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            int step = 0;
            for (int t = pair; t < tiles; t += pairs) {
                const int rb = t / col_blocks, cb = t - rb * col_blocks;
                const int arow = rb * 2 * GB_ROWS + rank * GB_ROWS, brow = cb * GP_NC + rank * GP_HALF;
                bool ok = true;
                for (int ks = 0; ks < ksteps; ks++, step++) {
                    const int s = step % S;
                    if (!gb_bar_wait(gb_smem(&bars.empty[s]), ((uint32_t)(step / S) & 1u) ^ 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    const uint32_t own = gb_smem(&bars.full[s]), bar = gp_of_rank(own, 0), stage = smem + (uint32_t)(s * GP_STAGE);
                    if (rank == 0) gb_bar_expect(own, 2 * GP_STAGE);
                    gp_tma_load(stage, &wmap, ks * GB_K, arow, bar);
                    gp_tma_load(stage + GP_A_BYTES, &xmap, ks * GB_K, brow, bar);
                }
                if (!ok) break;
            }
            // the copies in flight, also when this CTA gave up: the stages they fill come free (bounded) only after they have landed
            for (int p = step; p < step + S; p++) {
                for (uint32_t it = 0; it < GB_WAIT_LIMIT; it++) {
                    uint32_t ok;
                    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                                 : "=r"(ok) : "r"(gb_smem(&bars.empty[p % S])), "r"(((uint32_t)(p / S) & 1u) ^ 1u) : "memory");
                    if (ok) break;
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            int step = 0, j = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, j++) {
                const int ts = j % GB_TSTAGES;
                if (!gb_bar_wait(gb_smem(&bars.tempty[ts]), ((uint32_t)(j / GB_TSTAGES) & 1u) ^ 1u, abort_flag)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_acc = tmem + (uint32_t)(ts * GP_NC);
                for (int ks = 0; ks < ksteps; ks++, step++) {
                    const int s = step % S;
                    if (!gb_bar_wait(gb_smem(&bars.full[s]), (uint32_t)(step / S) & 1u, abort_flag)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t stage = smem + (uint32_t)(s * GP_STAGE);
                    const uint64_t ad = gb_desc(stage), bd = gb_desc(stage + GP_A_BYTES);
#pragma unroll
                    for (int i = 0; i < GB_K / 16; i++) gp_mma(d_acc, ad + 2 * i, bd + 2 * i, GP_IDESC, (ks | i) != 0);   // 32 bytes on per K = 16
                    gp_commit(gb_smem(&bars.empty[s]));
                }
                if (ok) gp_commit(gb_smem(&bars.tfull[ts]));
            }
        }
    } else if (warp >= GB_EPI_WARP0) {
        const int q = warp & 3, h = (warp - GB_EPI_WARP0) >> 2;   // tensor-memory lanes 32 q .., first or second half of the columns
        int j = 0;
        for (int t = pair; t < tiles; t += pairs, j++) {
            const int rb = t / col_blocks, cb = t - rb * col_blocks, ts = j % GB_TSTAGES;
            if (!__all_sync(0xffffffffu, gb_bar_wait(gb_smem(&bars.tfull[ts]), (uint32_t)(j / GB_TSTAGES) & 1u, abort_flag))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = rb * 2 * GB_ROWS + rank * GB_ROWS + 32 * q + lane, col0 = cb * GP_NC;
            const uint32_t trow = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(ts * GP_NC);
            const uint32_t free_bar = gp_of_rank(gb_smem(&bars.tempty[ts]), 0);
            gb_drain(o, trow, row, col0, GP_HALF * h, GP_HALF * h + GP_HALF, [&] {
                if (lane == 0) gp_arrive(free_bar);
            });
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gp_cluster_sync();   // nothing of either CTA reaches into the other any more
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GB_TSTAGES * GP_NC) : "memory");
    }
    if (threadIdx.x == 0 && bars.abort_flag) atomicExch(err, GB_ERR_WAIT);
}

template <int NC>
int launch_nc(const DenseMm &d, int sms, cudaStream_t s) {
    using C = GbCfg<NC>;
    static bool attr_done[64] = {false};
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    B200_REQUIRE(dev >= 0 && dev < 64, "gemm: device index %d out of range", dev);
    if (!attr_done[dev]) {
        B200_CUDA(cudaFuncSetAttribute(gemm_bf16_tcgen05_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        attr_done[dev] = true;
    }
    CUtensorMap wmap, xmap;
    int rc = rows_map(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.w, d.k, d.n, d.ldw, GB_ROWS);
    if (rc == B200_STATUS_SUCCESS) rc = rows_map(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.x, d.k, d.m, d.ldx, NC);
    if (rc != B200_STATUS_SUCCESS) return rc;
    int *err = nullptr;
    rc = device_error_word(&err);
    if (rc != B200_STATUS_SUCCESS) return rc;
    const int64_t rb = (d.n + GB_ROWS - 1) / GB_ROWS, cb = (d.m + NC - 1) / NC;
    B200_REQUIRE(rb * cb < (1ll << 31), "gemm: too many tiles");
    const GbOut o = {d.y, d.y_type, d.ldy, d.addend, d.ld_addend, d.bias, d.act, d.act_limit, d.act_alpha, (int)d.n, (int)d.m};
    const int tiles = (int)(rb * cb);
    return launch_pdl(gemm_bf16_tcgen05_kernel<NC>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(GB_THREADS), (size_t)C::SMEM, s, wmap, xmap, o,
                      (int)((d.k + GB_K - 1) / GB_K), (int)cb, tiles, err);
}

int launch_pair(const DenseMm &d, int sms, cudaStream_t s) {
    static bool attr_done[64] = {false};
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    B200_REQUIRE(dev >= 0 && dev < 64, "gemm: device index %d out of range", dev);
    if (!attr_done[dev]) {
        B200_CUDA(cudaFuncSetAttribute(gemm_bf16_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM));
        attr_done[dev] = true;
    }
    CUtensorMap wmap, xmap;
    int rc = rows_map(&wmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.w, d.k, d.n, d.ldw, GB_ROWS);
    if (rc == B200_STATUS_SUCCESS) rc = rows_map(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, d.x, d.k, d.m, d.ldx, GP_HALF);
    if (rc != B200_STATUS_SUCCESS) return rc;
    int *err = nullptr;
    rc = device_error_word(&err);
    if (rc != B200_STATUS_SUCCESS) return rc;
    const int64_t rb = (d.n + 2 * GB_ROWS - 1) / (2 * GB_ROWS), cb = (d.m + GP_NC - 1) / GP_NC;
    B200_REQUIRE(rb * cb < (1ll << 30), "gemm: too many tiles");
    const GbOut o = {d.y, d.y_type, d.ldy, d.addend, d.ld_addend, d.bias, d.act, d.act_limit, d.act_alpha, (int)d.n, (int)d.m};
    const int tiles = (int)(rb * cb), pairs = tiles < sms / 2 ? tiles : sms / 2;
    return launch_pdl_cluster(gemm_bf16_pair_kernel, dim3((unsigned)(2 * pairs)), dim3(GP_THREADS), 2u, (size_t)GP_SMEM, s, wmap, xmap, o,
                              (int)((d.k + GB_K - 1) / GB_K), (int)cb, tiles, err);
}

}  // namespace

// what the tensor maps can describe: 16-byte aligned bases and row strides
bool gemm_bf16_takes(const DenseMm &d) {
    return d.w_type == B200_TYPE_BF16 && d.x_type == B200_TYPE_BF16 && d.k % 8 == 0 && d.ldx % 8 == 0 && d.ldw % 8 == 0 && (((uintptr_t)d.w | (uintptr_t)d.x) & 15) == 0 &&
           d.n < (1ll << 31) - 256 && d.m < (1ll << 31) - 256 && d.norm_w == nullptr;
}

// Which form takes n weight rows x m activation rows: the activation rows of a CTA's tile (64, 128, 256), or 2 for pairs.  Each form by its waves
// times what one takes: a 128 x 128 tile as 5 per element of K, a pair's 256 x 256 one 6 (half the MMA time of its four quarters and as many
// copies as one of them), a 128 x 256 one 7; with short rows the drain (800 elements' worth; four warps over 256 columns 1100).  us as 128 x 128,
// 128 x 256 and pairs, waves in brackets, K 4096: 11008 x 300 rows 45 (2), 54 (2), 48 (2); 4096 x 2048 85 (4), 55 (2), 50 (2); K 2048: 6272 x 700 27 (2),
// 20 (1), 28 (2); 8192 x 2048 77 (7), 61 (4), 55 (4); K 512: 6272 x 3000 37 (8), 35 (4), 32 (5).
// A pair also starts a microsecond later (cluster, tensor memory of both SMs), which one wave of short rows and a column block filled to
// 160 of its 256 rows at most does not make up: 12288 x 2048 on 140 rows 16.7, 17.3 as pairs; on 192 17.9, 17.7; 12288 x 4096 on 140 31.1, 28.8
int gemm_bf16_pick_for(int64_t n, int64_t k, int64_t m, int sms) {
    if (m <= 64) return 64;
    if (m <= 128) return 128;
    const auto waves = [&](int64_t rows, int64_t cols, int64_t at_once) { return (((n + rows - 1) / rows) * ((m + cols - 1) / cols) + at_once - 1) / at_once; };
    const int64_t w128 = waves(GB_ROWS, 128, sms), w256 = waves(GB_ROWS, 256, sms), wp = sms > 1 ? waves(2 * GB_ROWS, GP_NC, sms / 2) : INT32_MAX;
    if (w128 > 1 && w256 == 1 && wp == 1 && m <= 160 && k <= 2048) return 256;
    const int64_t short_k = k < 800 ? 800 : k, t128 = 5 * w128 * short_k, t256 = 7 * w256 * (k < 1100 ? 1100 : k), tp = 6 * wp * short_k;
    return t128 <= t256 && t128 <= tp ? 128 : tp <= t256 ? 2 : 256;
}

int launch_gemm_bf16(const DenseMm &d, cudaStream_t s) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    switch (gemm_bf16_pick_for(d.n, d.k, d.m, sms)) {
        case 64: return launch_nc<64>(d, sms, s);
        case 128: return launch_nc<128>(d, sms, s);
        case 256: return launch_nc<256>(d, sms, s);
        default: return launch_pair(d, sms, s);
    }
}

}  // namespace b200
