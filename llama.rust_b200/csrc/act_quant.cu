// On-the-fly Q8 quantization of f32 activation rows, bit-exact with the CPU
// path's three value rules:
//   A1 quantize_row_q8_0      crates/ggml/src/quants.rs:331-362
//   A2 quantize_row_q8_K      crates/ggml/src/quants.rs:615-654
//   A3 quantize_mat_q8_K_4x8  crates/ggml/src/repack.rs:1561-1606 (values; the
//      4-row interleaved storage is a CPU detail, the device keeps plain rows)
// Every float op is an explicit round-to-nearest intrinsic: no FMA contraction.
#include "common.cuh"
#include "act_quant.cuh"

namespace b200 {

static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

size_t act_scratch_bytes(int64_t m, int64_t k) {
    size_t b = 0;
    b += align_up((size_t)m * k, 256);            // qs
    b += align_up((size_t)m * (k / 256) * 4, 256);  // d
    b += align_up((size_t)m * (k / 16) * 2, 256);   // bsums
    b += align_up((size_t)m * (k / 32) * 2, 256);   // dh
    return b;
}

ActBuf act_carve(void *scratch, int64_t m, int64_t k) {
    uint8_t *p = (uint8_t *)scratch;
    ActBuf a;
    a.k = k;
    a.qs = (int8_t *)p;
    p += align_up((size_t)m * k, 256);
    a.d = (float *)p;
    p += align_up((size_t)m * (k / 256) * 4, 256);
    a.bsums = (int16_t *)p;
    p += align_up((size_t)m * (k / 16) * 2, 256);
    a.dh = (uint16_t *)p;
    return a;
}

size_t act_f16_bytes(int64_t m, int64_t k) {
    if (m < ACT_F16_MIN_ROWS || k % GROUP_K != 0) return 0;
    return align_up((size_t)m * k * 2, 256) + (size_t)(k / 32) * align_up((size_t)m, 128) * 4;
}

ActF16 act_f16_carve(void *block, int64_t m, int64_t k) {
    ActF16 a;
    if (block == nullptr || act_f16_bytes(m, k) == 0) return a;
    a.x = (uint16_t *)block;
    a.scales = (float *)((uint8_t *)block + align_up((size_t)m * k * 2, 256));
    a.ld = (int64_t)align_up((size_t)m, 128);   // whole column blocks of the kernel's widest tile
    return a;
}

// A2 / A3: one CTA of 256 threads per (256-element block, row); the block's arithmetic is q8_K_block_store
// (act_quant.cuh), shared with the kernels that quantize what they have just computed.
template <bool A3>
__global__ void __launch_bounds__(256) quantize_q8_K_kernel(const float *__restrict__ x, int64_t ldx, ActBuf out) {
    pdl_trigger();
    pdl_wait();   // x comes from the previous kernel; the scratch written here may still be read by it
    const int64_t blk = blockIdx.x, row = blockIdx.y;
    q8_K_block_store<A3>(x[row * ldx + blk * 256 + threadIdx.x], out, row, blk);
}

// The same for prompt batches (more than 32 rows): one warp per block, lane l holding elements 8 l .. 8 l + 7, no
// CTA barrier (q8_K_block_store_warp); 16-byte loads when the rows allow it.
template <bool A3>
__global__ void __launch_bounds__(256) quantize_q8_K_rows_kernel(const float *__restrict__ x, int64_t ldx, ActBuf out, int nblk, int64_t nwork, bool vec) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int64_t wg = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (wg >= nwork) return;
    const int64_t row = wg / nblk, blk = wg - row * nblk;
    const float *p = x + row * ldx + blk * 256 + 8 * lane;
    float v[8];
    if (vec) {
        const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = p[j];
    }
    q8_K_block_store_warp<A3>(v, out, row, blk);
}

template <bool A3>
static int launch_q8_K(int64_t m, int64_t k, const float *x, int64_t ldx, ActBuf out, cudaStream_t s) {
    if (m <= 32) return launch_pdl(quantize_q8_K_kernel<A3>, dim3((unsigned)(k / 256), (unsigned)m), dim3(256), 0, s, x, ldx, out);
    const int64_t nblk = k / 256, nwork = nblk * m, blocks = (nwork + 7) / 8;
    B200_REQUIRE(blocks < 0x7fffffffLL, "quantize q8_K: tensor too large for one launch");
    const bool vec = ((uintptr_t)x & 15) == 0 && ldx % 4 == 0;
    return launch_pdl(quantize_q8_K_rows_kernel<A3>, dim3((unsigned)blocks), dim3(256), 0, s, x, ldx, out, (int)nblk, nwork, vec);
}

__device__ __forceinline__ float q8_0_scale(float amax) { return __fdiv_rn(amax, 127.0f); }
__device__ __forceinline__ float q8_0_inverse(float amax) { return amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f; }
__device__ __forceinline__ int q8_0_quant(float v, float id) {
    const float r = rintf(__fmul_rn(v, id));
    if (isnan(r) || fabsf(r) >= 2147483648.0f) return -128;  // the AVX2 cvt/packs saturation
    return max(-128, min(127, (int)r));
}
// A1: one warp per 32-element block, 8 blocks per CTA.
__global__ void __launch_bounds__(256) quantize_q8_0_kernel(const float *__restrict__ x, int64_t ldx, ActBuf out) {
    pdl_trigger();
    pdl_wait();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int64_t row = blockIdx.y;
    const int64_t blk = (int64_t)blockIdx.x * 8 + warp;
    if (blk >= out.k / 32) return;
    const float v = x[row * ldx + blk * 32 + lane];
    float amax = fabsf(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    out.qs[row * out.k + blk * 32 + lane] = (int8_t)q8_0_quant(v, q8_0_inverse(amax));
    if (lane == 0) out.dh[row * (out.k / 32) + blk] = __half_as_ushort(__float2half_rn(q8_0_scale(amax)));
}
// The same with the f16 form beside it: a CTA takes 8 rows (a warp each) x 256 elements, a thread 8 elements of a block, so that the f32 scales
// of neighbouring rows meet in a sector.  Rows from m on: zero scales
__global__ void __launch_bounds__(256) quantize_q8_0_f16_kernel(const float *__restrict__ x, int64_t ldx, ActBuf out, ActF16 f16, int64_t m, bool vec) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.y * 8 + (threadIdx.x >> 5), at = (int64_t)blockIdx.x * 256 + 8 * lane, blk = at / 32;
    if (row >= m) {
        if ((lane & 3) == 0 && row < f16.ld) f16.scales[blk * f16.ld + row] = 0.0f;
        return;
    }
    const float *p = x + row * ldx + at;
    float v[8];
    if (vec) {
        const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = p[j];
    }
    float amax = fabsf(v[0]);
#pragma unroll
    for (int j = 1; j < 8; j++) amax = fmaxf(amax, fabsf(v[j]));
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float id = q8_0_inverse(amax);
    int q[8];
#pragma unroll
    for (int j = 0; j < 8; j++) q[j] = q8_0_quant(v[j], id);
    const auto bytes = [](int a, int b, int c, int d) { return (uint32_t)(a & 0xff) | (uint32_t)(b & 0xff) << 8 | (uint32_t)(c & 0xff) << 16 | (uint32_t)(d & 0xff) << 24; };
    const auto halves = [](int a, int b) { return (uint32_t)__half_as_ushort(__int2half_rn(a)) | (uint32_t)__half_as_ushort(__int2half_rn(b)) << 16; };
    *reinterpret_cast<uint2 *>(out.qs + row * out.k + at) = make_uint2(bytes(q[0], q[1], q[2], q[3]), bytes(q[4], q[5], q[6], q[7]));
    *reinterpret_cast<uint4 *>(f16.x + row * out.k + at) = make_uint4(halves(q[0], q[2]), halves(q[1], q[3]), halves(q[4], q[6]), halves(q[5], q[7]));
    if ((lane & 3) == 0) {
        const __half d = __float2half_rn(q8_0_scale(amax));
        out.dh[row * (out.k / 32) + blk] = __half_as_ushort(d);
        f16.scales[blk * f16.ld + row] = __half2float(d);
    }
}

int launch_quantize_acts(int kind, int64_t m, int64_t k, const float *x, int64_t ldx, ActBuf out, cudaStream_t s, ActF16 f16) {
    B200_REQUIRE(m >= 0 && m <= 65535, "quantize: %lld activation rows exceed one launch (max 65535)", (long long)m);
    if (m == 0) return B200_STATUS_SUCCESS;
    if (kind == B200_ACT_Q8_0) {
        B200_REQUIRE(k > 0 && k % 32 == 0, "quantize q8_0: k = %lld must be a positive multiple of 32", (long long)k);
        if (f16.x) {
            const bool vec = ((uintptr_t)x & 15) == 0 && ldx % 4 == 0;
            return launch_pdl(quantize_q8_0_f16_kernel, dim3((unsigned)(k / 256), (unsigned)(f16.ld / 8)), dim3(256), 0, s, x, ldx, out, f16, m, vec);
        }
        dim3 grid((unsigned)((k / 32 + 7) / 8), (unsigned)m);
        return launch_pdl(quantize_q8_0_kernel, grid, dim3(256), 0, s, x, ldx, out);
    } else if (kind == B200_ACT_Q8_K || kind == B200_ACT_Q8_K_4X8) {
        B200_REQUIRE(k > 0 && k % 256 == 0, "quantize q8_K: k = %lld must be a positive multiple of 256", (long long)k);
        if (kind == B200_ACT_Q8_K) return launch_q8_K<false>(m, k, x, ldx, out, s);
        return launch_q8_K<true>(m, k, x, ldx, out, s);
    } else if (kind == B200_ACT_Q8_K_MIXED) {
        B200_REQUIRE(k > 0 && k % 256 == 0, "quantize q8_K: k = %lld must be a positive multiple of 256", (long long)k);
        const int64_t m4 = m - m % 4;
        if (m4 > 0) {
            int rc = launch_q8_K<true>(m4, k, x, ldx, out, s);
            if (rc != B200_STATUS_SUCCESS) return rc;
        }
        if (m > m4) {
            ActBuf tail = out;
            tail.qs += m4 * k;
            tail.d += m4 * (k / 256);
            tail.bsums += m4 * (k / 16);
            int rc = launch_q8_K<false>(m - m4, k, x + m4 * ldx, ldx, tail, s);
            if (rc != B200_STATUS_SUCCESS) return rc;
        }
    } else {
        B200_REQUIRE(false, "quantize: unknown activation kind %d", kind);
    }
    B200_CUDA(cudaGetLastError());
    return B200_STATUS_SUCCESS;
}

}  // namespace b200
