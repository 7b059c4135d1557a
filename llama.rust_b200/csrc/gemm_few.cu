// Mat-muls of a few activation rows (2 and more: batched decode steps, short prompts, routed experts) under the fast numerics policy, all five
// weight types.
//
// With few columns a mat-mul is a walk through the weights, so everything is laid out for that walk.  A CTA takes 8 or 16 activation rows and goes
// from row tile to row tile (32 weight rows each), its warps sharing the tile's K: a warp takes whole (tile, 256-element group) chunks, one bulk
// copy each into slots of its own in shared memory, the next chunk (of the next tile, too) asked for as soon as a slot is free, the first
// ones before the previous kernel in the stream has finished.  With 4-bit weights 74 KB of a CTA are on their way, and a SM has two.
// A chunk's bytes become the A fragments of mma.sync m16n8k32 (s8) in registers; the activations come from L2 as whole pieces, half a group at
// a time and one half ahead, through a few rows of shared memory of the warp's own.  No unpacked weight is ever written anywhere.  Sums of
// warps, and of a pair of CTAs that share a tile's K where there are few tiles, are added in a fixed order through shared memory.
// (mma.sync and not tcgen05: operands of 16 columns leave the tensor core idle either way, and this one takes them from registers.)
//   Q4_K, Q6_K: a sub-block's exact integer dots times its integer scale are added up as integers over the whole super-block, the mins of
//   Q4_K as one f16 product of the 6-bit mins with the activations' 16-element sums (both exact in f16, the sum exact in f32); one f32 fma
//   per super-block, where the exact kernels' chains take four or eight.
//   Q8_0, Q4_0, MXFP4: the exact integer dot of each 32-element block times d_w d_x (exact in f32 for f16 scales), added in f32; the dot comes
//   out of the product as a float already (the accumulator starts at the bits of 1.5 * 2^23).
// Every output is within a few f32 roundings of the exact sum over the quantized operands: from float64, of the result's norm, at K = 2048, 4096 and
// 14336, Q4_K 9e-8 / 9e-8 / 1.0e-7 where the chains it stands in for are 3e-7 / 4.5e-7 / 9e-7, Q6_K 5.4e-8 / 6.1e-8 / 6.8e-8 (5.8e-8 / 7.8e-8 / 1.4e-7),
// Q8_0 and Q4_0 7e-8 / 8e-8 / 1.1e-7 (1.4e-7 / 2.0e-7 / 3.8e-7), MXFP4 6e-8 / 6e-8 / 9e-8 (1.1e-7 / 1.8e-7 / 3.6e-7).  (Q6_K short rows: added up warp
// after warp, and with a super-block's product rounded before it meets the activation's scale, they were 6.5e-8.)
// What was tried: 32 columns per CTA (128 registers: spills; 255: one CTA per SM; both slower than two passes of 16 columns), a warp per tile in place
// of shared tiles (no change), 8-byte activation fragments straight from L2 (slower by a tenth at 16 columns), a CTA per tile without the
// walk (28672 x 4096 on 16 rows 30 us; with it 27), scales fetched byte by byte.  Figures against the other kernels: at few_takes below.
// Waits are bounded: one that runs out records error code 4, and its CTA (and the other of a pair) stores neither that tile nor a later one of its
// walk, and ends once its own copies have landed.
#include <algorithm>
#include <cstdlib>

#include "common.cuh"

namespace b200 {

namespace {

constexpr int FEW_WARPS = 8, FEW_THREADS = FEW_WARPS * 32, FEW_PITCH = 36;   // floats of a column's 32 partial sums: fragments fall on different banks
constexpr unsigned FEW_SPIN = 1u << 20;   // polls that sleep up to a microsecond each
constexpr int FEW_ERR_WAIT = 4;
constexpr int FEW_MAGIC = 0x4B400000;     // 1.5 * 2^23: adding an integer below 2^22 to these bits adds it to the float

template <int TYPE> struct FewType;
template <> struct FewType<B200_TYPE_Q4_K> { static constexpr int CHUNK = 4608, SLOTS = 2; };
template <> struct FewType<B200_TYPE_Q6_K> { static constexpr int CHUNK = 6720, SLOTS = 1; };
template <> struct FewType<B200_TYPE_Q8_0> { static constexpr int CHUNK = 8704, SLOTS = 1; };
template <> struct FewType<B200_TYPE_Q4_0> { static constexpr int CHUNK = 4608, SLOTS = 2; };
template <> struct FewType<B200_TYPE_MXFP4> { static constexpr int CHUNK = 4352, SLOTS = 2; };

struct FewArgs {
    const uint8_t *tiles[3];
    float *dst[3];
    int64_t n[3], lddst[3];
    int tile_start[4];       // matrix e owns row tiles tile_start[e] .. tile_start[e + 1] of the launch
    ActView acts;
    int64_t m;
    int nb, splits, col_blocks, walkers;
    GroupMap gm;             // work_expert set: column blocks are the experts' work items
    int *err;
    unsigned spin;           // polls of a wait
    int skip;                // test hook: the unit that the first warp of the first CTA does not ask for, -1: none
};

__device__ __forceinline__ uint32_t few_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// a warp's: the same answer for every lane
__device__ __forceinline__ bool few_wait(uint32_t bar, unsigned parity, unsigned spin) {
    unsigned ok = 0;
    for (unsigned i = 0; i < spin && !ok; i++)
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(bar), "r"(parity), "r"(1000u) : "memory");
    return __all_sync(0xffffffffu, ok != 0);
}
__device__ __forceinline__ void few_bulk(uint32_t dst, const void *src, unsigned bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void few_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, int c) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void few_mma16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ void few_mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ uint64_t few_pair(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t few_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t few_mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t few_add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// the integers 0 .. 63 in two bytes of x as f16
__device__ __forceinline__ uint32_t few_byte_f16x2(uint32_t x, uint32_t selector) {
    const uint32_t h = __byte_perm(x, 0x64646464u, selector);   // 1024 + byte
    const __half2 r = __hsub2(*(const __half2 *)&h, __half2half2(__ushort_as_half(0x6400)));
    return *(const uint32_t *)&r;
}
__device__ __forceinline__ uint32_t few_short_f16x2(uint32_t x) {
    const __half2 r = __halves2half2(__short2half_rn((short)(x & 0xffffu)), __short2half_rn((short)(x >> 16)));
    return *(const uint32_t *)&r;
}

// four 8 x 16-byte matrices whose rows the lanes point at: lane (g8, t) gets bytes 4 t .. 4 t + 3 of row g8 of each, which is what a lane supplies
// of a 16-element half of a sub-block
__device__ __forceinline__ void few_ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

constexpr int FEW_XPITCH = 144;   // bytes of a staged activation row of 128 elements: the eight rows of a fragment fall on different banks

// what a warp keeps of a chunk while it goes through its two halves.  Lane (g8, t) = (lane / 4, lane % 4) holds weight rows 16 mt + g8 and + 8
// (index r) and the sums of columns 8 nt + 2 t and + 1
template <int TYPE, int NT, bool GROUPED>
struct FewChunk {
    static constexpr bool KQ = TYPE == B200_TYPE_Q4_K || TYPE == B200_TYPE_Q6_K;
    int ig[KQ ? 2 : 1][KQ ? NT : 1][4];
    float dx[NT];        // K-quants: the scale of activation row 8 nt + g8
    uint32_t bs[NT][2];  // Q4_K: its 16-element sums 2 t, 2 t + 1 and 2 t + 8, 2 t + 9
    uint4 dh[NT];        // the others: its eight f16 scales
    uint32_t sc[TYPE == B200_TYPE_Q4_K ? 2 : 1][2][2];   // Q4_K: the eight 6-bit scales of a row, one per byte (crates/ggml/src/quants.rs:421-429)

    // xb: index of an activation row's first super-block
    __device__ __forceinline__ void begin(const ActView &acts, const uint32_t (&xb)[NT], int b) {
        const int t = threadIdx.x & 3;
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const uint32_t at = xb[nt] + (uint32_t)b;
            if (KQ) dx[nt] = acts.d[at];
            else dh[nt] = *((const uint4 *)acts.dh + at);
            if (TYPE == B200_TYPE_Q4_K) {
                const uint32_t *p = (const uint32_t *)acts.bsums + (uint64_t)at * 8 + t;
                bs[nt][0] = p[0];
                bs[nt][1] = p[4];
            }
        }
        if (KQ) {
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
                for (int nt = 0; nt < NT; nt++)
#pragma unroll
                    for (int e = 0; e < 4; e++) ig[KQ ? mt : 0][KQ ? nt : 0][e] = 0;
        }
    }

    // activation fragments of 32-element block j of the staged half: y[nt][first, second 16 elements]
    __device__ __forceinline__ static void columns(uint32_t stage, int j, uint32_t (&y)[NT][2]) {
        const int lane = threadIdx.x & 31;
        if (NT == 1) {
            uint32_t r[2];
            asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                         : "=r"(r[0]), "=r"(r[1]) : "r"(stage + (lane & 7) * FEW_XPITCH + 32 * j + ((lane >> 3) & 1) * 16) : "memory");
            y[0][0] = r[0];
            y[0][1] = r[1];
        } else {
#pragma unroll
            for (int nt = 0; nt < NT; nt += 2) {
                uint32_t r[4];
                few_ldsm4(r, stage + (8 * nt + (lane & 7) + ((lane >> 4) << 3)) * FEW_XPITCH + 32 * j + ((lane >> 3) & 1) * 16);
                y[nt][0] = r[0];
                y[nt][1] = r[1];
                y[nt + (NT > 1)][0] = r[2];
                y[nt + (NT > 1)][1] = r[3];
            }
        }
    }

    // half h (128 elements) of the chunk at w in shared memory against the staged half rows
    __device__ __forceinline__ void half(const uint8_t *w, uint32_t stage, int h, int nt_live, uint64_t (&acc)[2][NT][2]) {
        const int lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
        const uint32_t rows = few_smem(w) + lane * 16;   // a 512-byte piece of the chunk is 32 rows x 16 bytes
        if (TYPE == B200_TYPE_Q4_K) {
            if (h == 0) {
#pragma unroll
                for (int mt = 0; mt < 2; mt++)
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        const uint4 x = *(const uint4 *)(w + (16 * mt + 8 * r + g8) * 16);
                        sc[TYPE == B200_TYPE_Q4_K ? mt : 0][r][0] = x.y & 0x3f3f3f3fu;
                        sc[TYPE == B200_TYPE_Q4_K ? mt : 0][r][1] = (x.w & 0x0f0f0f0fu) | (((x.y >> 6) & 0x03030303u) << 4);
                    }
            }
#pragma unroll
            for (int gg = 0; gg < 2; gg++) {
                const int g = 2 * h + gg;
                uint32_t lo[4], hi[4];   // bytes 0..15 and 16..31 of the pair's 32, rows g8, + 8, + 16, + 24
                few_ldsm4(lo, rows + 512 + (2 * g) * 512);
                few_ldsm4(hi, rows + 512 + (2 * g + 1) * 512);
#pragma unroll
                for (int u = 0; u < 2; u++) {   // sub-block 2 g + u: low or high nibbles
                    uint32_t y[NT][2];
                    columns(stage, 2 * gg + u, y);
#pragma unroll
                    for (int mt = 0; mt < 2; mt++) {
                        int s[2];
#pragma unroll
                        for (int r = 0; r < 2; r++) s[r] = (int)__byte_perm(sc[TYPE == B200_TYPE_Q4_K ? mt : 0][r][h], 0, 0x4440 + 2 * gg + u);
                        const uint32_t a0 = (lo[2 * mt] >> (4 * u)) & 0x0f0f0f0fu, a1 = (lo[2 * mt + 1] >> (4 * u)) & 0x0f0f0f0fu,
                                       a2 = (hi[2 * mt] >> (4 * u)) & 0x0f0f0f0fu, a3 = (hi[2 * mt + 1] >> (4 * u)) & 0x0f0f0f0fu;
#pragma unroll
                        for (int nt = 0; nt < NT; nt++) {
                            if (GROUPED && nt >= nt_live) continue;
                            int d[4];
                            few_mma(d, a0, a1, a2, a3, y[nt][0], y[nt][1], 0);
#pragma unroll
                            for (int e = 0; e < 4; e++) ig[KQ ? mt : 0][KQ ? nt : 0][e] += d[e] * s[e >> 1];
                        }
                    }
                }
            }
        } else if (TYPE == B200_TYPE_Q6_K) {
            uint2 s8[2][2];   // the half's eight int8 scales
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
                for (int r = 0; r < 2; r++) s8[mt][r] = *(const uint2 *)(w + 6144 + (16 * mt + 8 * r + g8) * 16 + 8 * h);
            uint32_t A[2][4], B[2][4], H[2][4];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                few_ldsm4(A[u], rows + (4 * h + u) * 512);
                few_ldsm4(B[u], rows + (4 * h + 2 + u) * 512);
                few_ldsm4(H[u], rows + 4096 + (2 * h + u) * 512);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint32_t y[NT][2];
                columns(stage, q, y);
#pragma unroll
                for (int u = 0; u < 2; u++) {   // sub-block of elements 128 h + 32 q + 16 u ..
                    uint32_t v[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const uint32_t x = q & 1 ? B[u][i] : A[u][i], hb = q == 0 ? H[u][i] << 4 : q == 1 ? H[u][i] << 2 : q == 2 ? H[u][i] : H[u][i] >> 2;
                        v[i] = ((q & 2 ? x >> 4 : x) & 0x0f0f0f0fu) | (hb & 0x30303030u);
                        v[i] = ((v[i] | 0x80808080u) - 0x20202020u) ^ 0x80808080u;   // minus 32, byte by byte
                    }
#pragma unroll
                    for (int mt = 0; mt < 2; mt++) {
                        int s[2];
#pragma unroll
                        for (int r = 0; r < 2; r++) s[r] = (int)(int8_t)((2 * q + u < 4 ? s8[mt][r].x : s8[mt][r].y) >> (8 * ((2 * q + u) & 3)));
#pragma unroll
                        for (int nt = 0; nt < NT; nt++) {
                            if (GROUPED && nt >= nt_live) continue;
                            int d[4];
                            few_mma16(d, v[2 * mt], v[2 * mt + 1], y[nt][u]);
#pragma unroll
                            for (int e = 0; e < 4; e++) ig[KQ ? mt : 0][KQ ? nt : 0][e] += d[e] * s[e >> 1];
                        }
                    }
                }
            }
        } else {
            uint2 ws[2][2];   // the half's four scales of the rows: f16 (MXFP4: bytes)
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int row = 16 * mt + 8 * r + g8;
                    if (TYPE == B200_TYPE_MXFP4) ws[mt][r].x = *(const uint32_t *)(w + 4096 + row * 8 + 4 * h);
                    else ws[mt][r] = *(const uint2 *)(w + (TYPE == B200_TYPE_Q8_0 ? 8192 : 4096) + row * 16 + 8 * h);
                }
            const uint64_t minus = few_pair(-__int_as_float(FEW_MAGIC), -__int_as_float(FEW_MAGIC));
#pragma unroll
            for (int p = 0; p < 2; p++) {   // blocks 4 h + 2 p and + 1
                uint64_t dx2[NT][2];
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    const uint32_t own = h == 0 ? (p == 0 ? dh[nt].x : dh[nt].y) : (p == 0 ? dh[nt].z : dh[nt].w);
                    const uint32_t u0 = __shfl_sync(0xffffffffu, own, 8 * t), u1 = __shfl_sync(0xffffffffu, own, 8 * t + 4);   // of columns 2 t and 2 t + 1
                    dx2[nt][0] = few_pair(f16_bits_to_f32((uint16_t)(u0 & 0xffffu)), f16_bits_to_f32((uint16_t)(u1 & 0xffffu)));
                    dx2[nt][1] = few_pair(f16_bits_to_f32((uint16_t)(u0 >> 16)), f16_bits_to_f32((uint16_t)(u1 >> 16)));
                }
#pragma unroll
                for (int o = 0; o < 2; o++) {
                    const int blk = 4 * h + 2 * p + o;
                    uint32_t y[NT][2], a0[4], a1[4];
                    columns(stage, 2 * p + o, y);
                    if (TYPE == B200_TYPE_Q8_0) {
                        few_ldsm4(a0, rows + (2 * blk) * 512);
                        few_ldsm4(a1, rows + (2 * blk + 1) * 512);
                    } else {
                        uint32_t v[4];
                        few_ldsm4(v, rows + blk * 512);
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            if (TYPE == B200_TYPE_MXFP4) {
                                mxfp4_values(v[i], &a0[i], &a1[i]);
                            } else {
                                a0[i] = (((v[i] & 0x0f0f0f0fu) | 0x80808080u) - 0x08080808u) ^ 0x80808080u;   // minus 8, byte by byte
                                a1[i] = ((((v[i] >> 4) & 0x0f0f0f0fu) | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
                            }
                        }
                    }
#pragma unroll
                    for (int mt = 0; mt < 2; mt++) {
                        uint64_t dw2[2];
#pragma unroll
                        for (int r = 0; r < 2; r++) {
                            const uint32_t word = p == 0 ? ws[mt][r].x : ws[mt][r].y;
                            const float dw = TYPE == B200_TYPE_MXFP4 ? e8m0_half_to_f32((ws[mt][r].x >> (8 * (2 * p + o))) & 0xffu) : f16_bits_to_f32((uint16_t)(o ? word >> 16 : word & 0xffffu));
                            dw2[r] = few_pair(dw, dw);
                        }
#pragma unroll
                        for (int nt = 0; nt < NT; nt++) {
                            if (GROUPED && nt >= nt_live) continue;
                            int d[4];
                            few_mma(d, a0[2 * mt], a0[2 * mt + 1], a1[2 * mt], a1[2 * mt + 1], y[nt][0], y[nt][1], FEW_MAGIC);
#pragma unroll
                            for (int r = 0; r < 2; r++)
                                acc[mt][nt][r] = few_fma2(few_add2(few_pair(__int_as_float(d[2 * r]), __int_as_float(d[2 * r + 1])), minus), few_mul2(dw2[r], dx2[nt][o]), acc[mt][nt][r]);
                        }
                    }
                }
            }
        }
    }

    // the super-block's integers into the sums
    __device__ __forceinline__ void end(const uint8_t *w, int nt_live, uint64_t (&acc)[2][NT][2]) {
        if (!KQ) return;
        const int lane = threadIdx.x & 31, g8 = lane >> 2, t = lane & 3;
        uint32_t mn[2][2][2];
        float dw[2][2], dm[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; mt++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int row = 16 * mt + 8 * r + g8;
                if (TYPE == B200_TYPE_Q4_K) {
                    const uint4 x = *(const uint4 *)(w + row * 16);
                    dw[mt][r] = f16_bits_to_f32((uint16_t)(x.x & 0xffffu));
                    dm[mt][r] = -f16_bits_to_f32((uint16_t)(x.x >> 16));
                    const uint32_t sel = 0x4040u | (uint32_t)t | (uint32_t)t << 8;   // 16-element sums 2 t, 2 t + 1 belong to sub-block t, 2 t + 8 and + 9 to t + 4
                    mn[mt][r][0] = few_byte_f16x2(x.z & 0x3f3f3f3fu, sel);
                    mn[mt][r][1] = few_byte_f16x2(((x.w >> 4) & 0x0f0f0f0fu) | (((x.z >> 6) & 0x03030303u) << 4), sel);
                } else {
                    dw[mt][r] = f16_bits_to_f32(*(const uint16_t *)(w + 6656 + row * 2));
                }
            }
        // Q6_K: what rounding a product leaves out is added first, where there is such a thing (asked for the warp: two selects a scale and activation
        // row took a 128256 x 4096 head on 16 rows from 143 to 159 us)
        bool finite = true;
        if (TYPE == B200_TYPE_Q6_K) {
            float far = fmaxf(fmaxf(fabsf(dw[0][0]), fabsf(dw[0][1])), fmaxf(fabsf(dw[1][0]), fabsf(dw[1][1])));
#pragma unroll
            for (int nt = 0; nt < NT; nt++) far = fmaxf(far, fabsf(dx[nt]));
            finite = !__any_sync(0xffffffffu, far == INFINITY);
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            if (GROUPED && nt >= nt_live) continue;
            const float d0 = __shfl_sync(0xffffffffu, dx[nt], 8 * t), d1 = __shfl_sync(0xffffffffu, dx[nt], 8 * t + 4);   // of columns 2 t and 2 t + 1
            const uint64_t dx2 = few_pair(d0, d1);
            uint32_t b0 = 0, b1 = 0;
            if (TYPE == B200_TYPE_Q4_K) {
                b0 = few_short_f16x2(bs[nt][0]);
                b1 = few_short_f16x2(bs[nt][1]);
            }
#pragma unroll
            for (int mt = 0; mt < 2; mt++) {
                float mg[4];
                if (TYPE == B200_TYPE_Q4_K) few_mma_f16(mg, mn[mt][0][0], mn[mt][1][0], mn[mt][0][1], mn[mt][1][1], b0, b1);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int *i2 = &ig[KQ ? mt : 0][KQ ? nt : 0][2 * r];
                    const uint64_t i2f = few_pair((float)i2[0], (float)i2[1]), d2 = few_pair(dw[mt][r], dw[mt][r]);
                    uint64_t v = few_mul2(i2f, d2);
                    if (TYPE == B200_TYPE_Q4_K) v = few_fma2(few_pair(mg[2 * r], mg[2 * r + 1]), few_pair(dm[mt][r], dm[mt][r]), v);
                    else if (finite) acc[mt][nt][r] = few_fma2(few_fma2(i2f, d2, v ^ 0x8000000080000000ull), dx2, acc[mt][nt][r]);
                    acc[mt][nt][r] = few_fma2(v, dx2, acc[mt][nt][r]);
                }
            }
        }
    }
};

template <int TYPE, int NT, bool GROUPED>
__global__ void __launch_bounds__(FEW_THREADS, 2)
gemm_few_kernel(const FewArgs a) {
    using T = FewType<TYPE>;
    // [warp][slot][chunk]; [warp][staged activations], at a tile's end its sums [warp][column][row]; [warp] the sums of its first class, likewise
    extern __shared__ __align__(128) uint8_t few_raw[];
    __shared__ uint64_t bars[FEW_WARPS * T::SLOTS];
    __shared__ int gave_up;   // for the other CTA of a pair
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)(blockIdx.x % (unsigned)a.splits), idx = (int)(blockIdx.x / (unsigned)a.splits);
    // row tiles first, first + walkers, .. of the launch, for one column block
    const int block = GROUPED ? idx / a.walkers : idx % a.col_blocks, first = GROUPED ? idx - block * a.walkers : idx / a.col_blocks;
    // A tile's groups in 16 classes, b % 16, each summed in order by one warp; an output is the sum, by halves, over w of (class w + class w + 8), whether
    // this CTA has all of them (a warp class w, then class w + 8) or the CTAs of a pair have eight each: the same bits either way
    const int c0 = warp + 8 * rank, n0 = c0 < a.nb ? (a.nb - 1 - c0) / 16 + 1 : 0;
    const int n1 = a.splits == 1 && warp + 8 < a.nb ? (a.nb - 9 - warp) / 16 + 1 : 0, mine = n0 + n1;
    const auto group = [&](int i) { return i < n0 ? c0 + 16 * i : warp + 8 + 16 * (i - n0); };
    const int units = mine * ((a.tile_start[3] - 1 - first) / a.walkers + 1);

    const uint32_t bar0 = few_smem(&bars[warp * T::SLOTS]);
    uint8_t *const slots = few_raw + warp * T::SLOTS * T::CHUNK;
    if (lane == 0) {
        for (int s = 0; s < T::SLOTS; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * s) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    int64_t expert = 0;
    if (GROUPED) {
        pdl_wait();
        // an item's columns in use come first: a block without any is done, as are the items past the last (every CTA of the cluster leaves: nothing has
        // been started yet)
        const int item = block / (4 / NT);
        if (item >= *a.gm.n_items || a.gm.col_act[(int64_t)block * (NT * 8)] < 0) return;
        expert = (int64_t)a.gm.work_expert[item] * a.gm.expert_bytes;
    }
    // lane 0 asks for the chunk of the warp's unit u: its group u % mine of the walk's tile u / mine
    int next_tile = first, next_group = 0;
    const auto ask = [&](int u) {
        const int me = next_tile >= a.tile_start[2] ? 2 : next_tile >= a.tile_start[1] ? 1 : 0;
        const uint8_t *src = a.tiles[me] + expert + ((int64_t)(next_tile - a.tile_start[me]) * a.nb + group(next_group)) * T::CHUNK;
        if (u != a.skip || (blockIdx.x | warp)) few_bulk(few_smem(slots + (u % T::SLOTS) * T::CHUNK), src, T::CHUNK, bar0 + 8 * (u % T::SLOTS));
        if (++next_group == mine) {
            next_group = 0;
            next_tile += a.walkers;
        }
    };
    if (lane == 0)
        for (int u = 0; u < T::SLOTS && u < units; u++) ask(u);
    if (!GROUPED) pdl_wait();   // the activations come from the previous kernel in the stream; the weights do not

    const int64_t col0 = (int64_t)block * (NT * 8);
    // activation rows: of column 8 nt + lane / 4 (its first super-block); of column 4 i + lane / 8, whose 16-byte pieces this lane stages (byte offset)
    uint32_t xb[NT], pieces[2 * NT];
    int nt_live = NT;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        const int64_t c = col0 + 8 * nt + (lane >> 2);
        int x;
        if (GROUPED) {
            x = a.gm.col_act[c];
            if (!__any_sync(0xffffffffu, x >= 0) && nt < nt_live) nt_live = nt;   // the columns in use come first
            if (x < 0) x = 0;
        } else {
            x = (int)(c < a.m ? c : a.m - 1);
            if (col0 + 8 * nt >= a.m && nt < nt_live) nt_live = nt;
        }
        xb[nt] = (uint32_t)x * (uint32_t)a.nb;
        pieces[2 * nt] = __shfl_sync(0xffffffffu, xb[nt], (lane >> 3) * 4) * GROUP_K + 16 * (lane & 7);
        pieces[2 * nt + 1] = __shfl_sync(0xffffffffu, xb[nt], (lane >> 3) * 4 + 16) * GROUP_K + 16 * (lane & 7);
    }
    // half h of group b of the activation rows, as 16-byte pieces
    uint4 xa[2 * NT];
    const auto fetch = [&](int b, int h) {
#pragma unroll
        for (int i = 0; i < 2 * NT; i++)
            if (!GROUPED || i < 2 * nt_live) xa[i] = *(const uint4 *)(a.acts.qs + (pieces[i] + (uint32_t)(b * GROUP_K + 128 * h)));
    };
    uint8_t *const stages = few_raw + FEW_WARPS * T::SLOTS * T::CHUNK, *const stage_g = stages + warp * (NT * 8 * FEW_XPITCH);
    const uint32_t stage = few_smem(stage_g);
    constexpr int PLANE = NT * 8 * FEW_PITCH;
    static_assert(PLANE * 4 == NT * 8 * FEW_XPITCH, "a warp's partial sums take the place of its staged activations");
    float *const red = (float *)stages, *const first_sums = red + FEW_WARPS * PLANE;
    if (mine) fetch(group(0), 0);
    bool ok = true;
    int u = 0;
    for (int g = first; g < a.tile_start[3]; g += a.walkers) {
        uint64_t acc[2][NT][2];
#pragma unroll
        for (int mt = 0; mt < 2; mt++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++) acc[mt][nt][0] = acc[mt][nt][1] = 0;
        // this lane's part of the warp's sums, into a plane [column][row]
        const auto put = [&](float *plane) {
#pragma unroll
            for (int mt = 0; mt < 2; mt++)
#pragma unroll
                for (int nt = 0; nt < NT; nt++)
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        float *p = plane + warp * PLANE + (8 * nt + 2 * (lane & 3)) * FEW_PITCH + 16 * mt + 8 * r + (lane >> 2);
                        p[0] = __uint_as_float((uint32_t)acc[mt][nt][r]);
                        p[FEW_PITCH] = __uint_as_float((uint32_t)(acc[mt][nt][r] >> 32));
                        acc[mt][nt][r] = 0;
                    }
        };
        for (int i = 0; i < mine && ok; i++, u++) {
            const int s = u % T::SLOTS;
            if (!few_wait(bar0 + 8 * s, (unsigned)(u / T::SLOTS) & 1u, a.spin)) {
                // No more copies are asked for, and those on their way are waited for, with a limit again.  The CTA walks on, for the barriers' sake,
                // and stores nothing any more
                if (lane == 0) atomicExch(a.err, FEW_ERR_WAIT);
                for (int j = 0; j < T::SLOTS && u + j < units; j++) few_wait(bar0 + 8 * ((u + j) % T::SLOTS), (unsigned)((u + j) / T::SLOTS) & 1u, a.spin);
                ok = false;
                break;
            }
            const uint8_t *w = slots + s * T::CHUNK;
            const int b = group(i);
            if (i == n0) put(first_sums);   // class w is done
            FewChunk<TYPE, NT, GROUPED> chunk;
            chunk.begin(a.acts, xb, b);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                __syncwarp();   // the stage has been read
#pragma unroll
                for (int v = 0; v < 2 * NT; v++) *(uint4 *)(stage_g + (4 * v + (lane >> 3)) * FEW_XPITCH + 16 * (lane & 7)) = xa[v];
                __syncwarp();
                if (h == 0) fetch(b, 1);
                else if (u + 1 < units) fetch(group(i + 1 < mine ? i + 1 : 0), 0);
                chunk.half(w, stage, h, nt_live, acc);
            }
            chunk.end(w, nt_live, acc);
            __syncwarp();
            if (lane == 0 && u + T::SLOTS < units) ask(u + T::SLOTS);
        }
        const int failed = __syncthreads_or(!ok);   // the staged activations have been read
        put(red);
        if (tid == 0) gave_up = failed;
        __syncthreads();
        const int me = g >= a.tile_start[2] ? 2 : g >= a.tile_start[1] ? 1 : 0;
        const int64_t row0 = (int64_t)(g - a.tile_start[me]) * TILE_ROWS, n = a.n[me], lddst = a.lddst[me];
        float *const dst = a.dst[me];
        const auto store = [&](int c, int row_in, float v) {
            const int64_t row = row0 + row_in;
            int64_t col = col0 + c;
            if (GROUPED) col = a.gm.col_out[col];
            if (row >= n || col < 0 || (!GROUPED && col >= a.m)) return;
            dst[col * lddst + row] = v;
            if (a.acts.sum) a.acts.sum[col * a.acts.ld_sum + row] = __fadd_rn(v, a.acts.addend[col * a.acts.ld_addend + row]);
        };
        const int w0 = a.nb < 8 ? a.nb : 8, w1 = a.nb - 8 < 8 ? a.nb - 8 : 8;   // classes that there are of the first and of the second eight
        if (a.splits == 1) {
            for (int i = tid; !failed && i < nt_live * 8 * 32; i += FEW_THREADS) {
                const int at = (i >> 5) * FEW_PITCH + (i & 31);
                float v[8];
#pragma unroll
                for (int p = 0; p < 8; p++) v[p] = p < w1 ? first_sums[p * PLANE + at] + red[p * PLANE + at] : p < w0 ? red[p * PLANE + at] : 0.0f;
                store(i >> 5, i & 31, ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
            }
            __syncthreads();   // the sums have been read: the next tile's activations may be staged
        } else {
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
            uint32_t p0, p1;   // the first and the second eight classes' sums
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p0) : "r"(few_smem(red)), "r"(0));
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p1) : "r"(few_smem(red)), "r"(1));
            uint32_t other;
            int other_failed;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(other) : "r"(few_smem(&gave_up)), "r"(rank ^ 1));
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(other_failed) : "r"(other) : "memory");
            for (int i = tid + rank * FEW_THREADS; !(failed | other_failed) && i < nt_live * 8 * 32; i += FEW_THREADS * 2) {
                const uint32_t at = (uint32_t)((i >> 5) * FEW_PITCH + (i & 31)) * 4;
                float x[16];
#pragma unroll
                for (int p = 0; p < 8; p++) {
                    x[2 * p] = x[2 * p + 1] = 0.0f;
                    if (p < w0) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x[2 * p]) : "r"(p0 + at + p * PLANE * 4) : "memory");
                    if (p < w1) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x[2 * p + 1]) : "r"(p1 + at + p * PLANE * 4) : "memory");
                }
                float v[8];
#pragma unroll
                for (int p = 0; p < 8; p++) v[p] = p < w1 ? x[2 * p] + x[2 * p + 1] : x[2 * p];
                store(i >> 5, i & 31, ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
            }
            // nobody's sums change or go while the other reads them
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }
}

// CTAs (a cluster) that share a tile's K: a pair where there are fewer tiles than about 1.4 per SM.  us, whole calls, 1 / 2 / 4 / 8 CTAs (Q4_K, 16 rows,
// each tile a CTA of its own): 14336 x 4096 16.6 / 24.6 / 34.7 / 63.8, 4096 x 14336 21.2 / 16.8 / 19.5 / 27.0, 1024 x 4096 on 32 rows
// 19.9 / 13.9 / 12.2 / 12.5.  More than a pair would need sums in another order: a matrix alone and one among its siblings give the same bits
int few_splits(int64_t ctas, int nb, int sms) { return ctas * 20 < (int64_t)sms * 27 && nb > 8 ? 2 : 1; }

// test hook: while a limit is set the waits poll that often, and a.skip is the unit of the first warp that is not asked for
unsigned g_few_spin = 0;
int g_few_skip = -1;

template <int TYPE, int NT, bool GROUPED>
int few_launch(FewArgs &a, int64_t column_blocks, int64_t live_blocks, int64_t act_rows, cudaStream_t s) {
    using T = FewType<TYPE>;
    constexpr size_t SMEM = (size_t)FEW_WARPS * (T::SLOTS * T::CHUNK + 2 * NT * 8 * FEW_XPITCH);
    static bool attr_done[64] = {false};
    static int sms[64] = {0};
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    B200_REQUIRE(dev >= 0 && dev < 64, "gemm: device index %d out of range", dev);
    if (!attr_done[dev]) {
        B200_CUDA(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev));
        B200_CUDA(cudaFuncSetAttribute(gemm_few_kernel<TYPE, NT, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
        attr_done[dev] = true;
    }
    B200_REQUIRE(act_rows * a.nb < FEW_ACT_GROUPS, "gemm few: %lld activation rows of %d super-blocks are too many", (long long)act_rows, a.nb);
    const int64_t tiles = a.tile_start[3];
    a.spin = g_few_spin ? g_few_spin : FEW_SPIN;
    a.skip = g_few_spin ? g_few_skip : -1;
    a.splits = few_splits(tiles * live_blocks, a.nb, sms[dev]);
    static_assert(SMEM * 2 + 4096 <= 227 * 1024, "two CTAs per SM");
    const int64_t slots = 2 * (int64_t)sms[dev];
    // walks over the row tiles: as many CTAs as run at once; of experts, whose number of items the host does not know, twice that
    const int64_t walkers = GROUPED ? (2 * slots + live_blocks - 1) / live_blocks : slots / (column_blocks * a.splits);
    a.walkers = (int)(walkers < 1 ? 1 : walkers < tiles ? walkers : tiles);
    const int64_t ctas = (int64_t)a.walkers * column_blocks * a.splits;
    B200_REQUIRE(ctas < 0x7fffffffLL, "gemm: %lld row tiles x %lld column blocks are too many for one launch", (long long)tiles, (long long)column_blocks);
    const dim3 grid((unsigned)ctas);
    if (a.splits == 1) return launch_pdl(gemm_few_kernel<TYPE, NT, GROUPED>, grid, dim3(FEW_THREADS), SMEM, s, a);
    return launch_pdl_cluster(gemm_few_kernel<TYPE, NT, GROUPED>, grid, dim3(FEW_THREADS), (unsigned)a.splits, SMEM, s, a);
}
template <int TYPE>
int few_launch_nt(FewArgs &a, int64_t m, cudaStream_t s) {
    a.col_blocks = (int)((m + 15) / 16);
    if (m <= 8) return few_launch<TYPE, 1, false>(a, 1, 1, m, s);
    return few_launch<TYPE, 2, false>(a, a.col_blocks, a.col_blocks, m, s);
}

}  // namespace

void gemm_few_debug_wait(int spin_limit, int skip_unit) {
    g_few_spin = spin_limit > 0 ? (unsigned)spin_limit : 0u;
    g_few_skip = skip_unit;
}

// Whether m activation rows are few, on a GPU of sms SMs.  us, weights from HBM, the others / this kernel:
//   * Up to 31 rows: 14336 x 4096 on 8 and 16 rows Q4_K 25 / 13 and 26 / 18, Q6_K 24 / 17 and 28 / 26, Q8_0 26 / 16 and 28 / 23, Q4_0 25 / 13 and
//     26 / 17, MXFP4 33 / 20 and 34 / 24; 4096 x 14336 Q8_0 73 / 18 and 75 / 22, on 4 rows 82 / 17.  But not Q6_K on 9 to 31 rows
//     of up to 8 super-blocks, where the exact kernel (gemm_mma.cu) is as quick or quicker: 6144 x 2048 on 20 12.4 / 14.4, 14336 x 2048 20 / 23.  (Of 16
//     it is a tenth quicker in small matrices, 4096 x 4096 on 12 rows 9.9 / 10.9, and slower in large ones, 128256 x 4096 on 16 158 / 145; 7.8e-8
//     from float64, 6.1e-8 here.)  One rule for every n: a matrix alone and one among its siblings take the same kernel.
//   * K-quants up to 63 rows: 14336 x 4096 on 48 Q4_K 66 / 39, Q6_K 69 / 54, 1000 x 2048 on 32 29 / 8.
//   * Above that by estimates, in microseconds, x = 10^6 weights, b = blocks of 16 rows: here 8 + c x b (instructions and waits for weights: a SM
//     issues in 38 to 44 % of its slots on 16 rows, and the weights are unpacked again for every block; more with less than 8 super-blocks, where warps have none), against
//       K-quants on the fast tcgen05 kernel (2048 weight rows and up, its rows in one block of 256): by its weights or, in few tiles, by its
//       latency a super-block, whichever says less;
//       K-quants of fewer weight rows, on the exact kernels: a latency a super-block too (one wave);
//       the others on int8 tiles of 128 x 32: 5 + 1.5 a wave and super-block, MXFP4 1.9, where the f16 kernel is not the better one.
//     The estimates are a little high for this kernel and low for the others: over 1190 products (n 512 to 32000, k 1024 to 14336, 32 to 512
//     rows, the five types) one that is taken is more than 3 % slower (6144 x 2048 Q4_K on 112 rows 23.6 / 24.5).  4096 x 14336 on 32 rows: Q4_K
//     118 / 24, Q6_K 189 / 35, Q8_0 95 / 28; 4096 x 4096 on 64: Q4_K 29 / 18, Q8_0 32 / 19; 1024 x 4096 Q6_K on 512 55 / 43.
bool few_takes_for(int type, int route, int64_t n, int64_t k, int64_t m, int sms) {
    if (m < 2 || n <= 0 || m * (k / GROUP_K) >= FEW_ACT_GROUPS) return false;   // 32-bit byte offsets into the activations
    const bool q6 = type == B200_TYPE_Q6_K, kq = type == B200_TYPE_Q4_K || q6;
    switch (type) {
        case B200_TYPE_Q4_K: break;
        case B200_TYPE_Q6_K:
            if (route != B200_ROUTE_TILED && route != B200_ROUTE_ROWDOT) return false;
            break;
        case B200_TYPE_Q8_0:
            if (route != B200_ROUTE_ROWDOT) return false;
            break;
        case B200_TYPE_Q4_0:
        case B200_TYPE_MXFP4:
            if (route != B200_ROUTE_REPACK) return false;
            break;
        default: return false;
    }
    if (q6 && route == B200_ROUTE_TILED && m > 8 && m < 32 && k <= 8 * GROUP_K) return false;
    if (m < 32 || (kq && m < GEMM_FAST_MIN_COLS)) return true;
    if (m > (kq && n >= 2048 ? 256 : 512)) return false;
    const double x = (double)n * (double)k * 1e-6 * 148 / sms, nb = (double)(k / GROUP_K), blocks = (double)((m + 15) / 16);   // per SM as on 148
    if (kq) {
        const double unpacking = (q6 ? 0.25 : 0.175) * x * blocks, here = 8.0 + unpacking + (nb < 8 ? unpacking * (8.0 / nb - 1.0) * 0.4 : 0.0);
        if (n < 2048) return here < 7.0 + (q6 ? 2.5 : 1.8) * nb;
        return here < std::min(20.0 + (q6 ? 0.80 : 0.40) * x, 9.0 + (q6 ? 2.4 : 1.9) * nb);
    }
    if (gemm_b32_pick_for(type, n, m, sms) != 0) return false;
    const int64_t waves = (((n + 127) / 128) * ((m + 31) / 32) + sms - 1) / sms;
    return 8.0 + (type == B200_TYPE_MXFP4 ? 0.25 : 0.182) * x * blocks < 5.0 + (type == B200_TYPE_MXFP4 ? 1.9 : 1.5) * nb * (double)waves;
}
// whether launch_gemv comes here: the fast numerics policy, and no switch for another kernel (B200_GEMM_FEW=0, B200_GEMM_FAST; read per call)
bool few_takes(int type, int route, int64_t n, int64_t k, int64_t m) {
    if (numerics_mode() != 1) return false;
    const char *e = getenv("B200_GEMM_FEW");
    if (e && e[0] == '0') return false;
    if (m >= GEMM_FAST_MIN_COLS && (type == B200_TYPE_Q4_K || type == B200_TYPE_Q6_K) && getenv("B200_GEMM_FAST")) return false;
    return few_takes_for(type, route, n, k, m, m < 32 ? 148 : sm_count());   // (of so few rows the number of SMs says nothing)
}
// MUL_MAT_ID, the pairs grouped by expert, by the pairs an expert has on average; us, the others / this kernel, even routing.
//   * Q6_K, Q8_0: the alternative reads an expert's weights once per pair.  From 4 pairs an expert on; 128 experts of 768 x 2048, 512 pairs 0.35 and
//     0.26 of its time.
//   * Q4_K: the same, but its per-pair kernel is quicker on rows of few super-blocks, of which most of this one's warps have none: 128 experts of
//     768 x 2048 on 512 pairs 68 / 45, 4096 pairs 502 / 135; 60 of 512 x 1024 on 256 pairs (4 each) 15 / 20, on 512 (8) 0.92; 256 x 512 2.1
//     times as long with 4 each, 1.5 with 8.
//   * MXFP4 and Q4_0 against int8 tiles of 128 rows x 32 pairs, up to 16 pairs an expert: 768 x 2048, 128 experts, 128 pairs 83 / 52 (64 / 39), 512 pairs
//     121 / 67 (92 / 50), 2048 pairs 0.91; 32 pairs an expert 174 / 189 (137 / 153).  Not rows of less than four super-blocks (256 x 512 1.1 to 1.5
//     times as long), with four to seven of them up to 4 pairs an expert only (512 x 1024, 60 experts of 8.5 pairs 1.0 to 1.08), and as few where
//     the int8 tiles are one wave (8 experts of 2048 x 2048, 128 pairs 1.17).  Routing as uneven as 1 / rank gains as much; where 8 of 128 experts have all
//     the pairs this kernel is up to a third slower, which the host cannot know.
bool few_takes_experts(int type, int64_t n, int64_t k, int64_t act_rows, int64_t n_expert, int64_t pairs) {
    if (numerics_mode() != 1 || pairs < 64 || pairs >= 0x7fffffffLL / 32 || n_expert >= (1 << 20) || act_rows * (k / GROUP_K) >= FEW_ACT_GROUPS) return false;
    const char *e = getenv("B200_GEMM_FEW");
    if (e && e[0] == '0') return false;
    const int64_t experts = n_expert < pairs ? n_expert : pairs, avg = pairs / experts, nb = k / GROUP_K;
    if (type == B200_TYPE_MXFP4 || type == B200_TYPE_Q4_0) return nb >= 4 && avg <= (nb < 8 || (n + 127) / 128 * experts <= sm_count() ? 4 : 16);
    if (type == B200_TYPE_Q4_K) return nb >= 4 && avg >= 4 && avg * nb >= 32;
    return avg >= 4;
}

// count matrices of one type and row length against the same m activation rows
int launch_gemm_few(int type, int count, const int64_t *n, int64_t k, int64_t m, const uint8_t *const *tiles, ActView acts, float *const *dst, const int64_t *lddst, cudaStream_t s) {
    B200_REQUIRE(k % GROUP_K == 0 && count >= 1 && count <= 3, "gemm few: bad shape");
    B200_REQUIRE(count == 1 || !acts.sum, "gemm: the fused add goes with a single matrix");
    FewArgs a = {};
    int64_t total = 0;
    for (int e = 0; e < 3; e++) {
        const int src = e < count ? e : count - 1;
        a.tiles[e] = tiles[src];
        a.dst[e] = dst[src];
        a.n[e] = n[src];
        a.lddst[e] = lddst[src];
        a.tile_start[e] = e < count ? (int)total : 0x7fffffff;
        if (e < count) total += (n[e] + TILE_ROWS - 1) / TILE_ROWS;
    }
    if (total == 0 || m == 0) return B200_STATUS_SUCCESS;
    B200_REQUIRE(total < 0x7fffffffLL, "gemm: %lld row tiles are too many for one launch", (long long)total);
    a.tile_start[3] = (int)total;
    a.acts = acts;
    a.m = m;
    a.nb = (int)(k / GROUP_K);
    const int rc = device_error_word(&a.err);
    if (rc != B200_STATUS_SUCCESS) return rc;
    switch (type) {
        case B200_TYPE_Q4_K: return few_launch_nt<B200_TYPE_Q4_K>(a, m, s);
        case B200_TYPE_Q6_K: return few_launch_nt<B200_TYPE_Q6_K>(a, m, s);
        case B200_TYPE_Q8_0: return few_launch_nt<B200_TYPE_Q8_0>(a, m, s);
        case B200_TYPE_Q4_0: return few_launch_nt<B200_TYPE_Q4_0>(a, m, s);
        case B200_TYPE_MXFP4: return few_launch_nt<B200_TYPE_MXFP4>(a, m, s);
        default: B200_REQUIRE(false, "gemm few: no kernel for weight type %d", type);
    }
}

// the experts' work items (32 columns each) of MUL_MAT_ID, in blocks of 8 or 16 columns by the pairs an expert has on average
template <int TYPE>
static int few_grouped(FewArgs &a, int64_t max_items, int64_t n_expert, int64_t pairs, int64_t act_rows, cudaStream_t s) {
    const int64_t experts = n_expert < pairs ? n_expert : pairs;
    if (pairs <= 4 * experts) return few_launch<TYPE, 1, true>(a, max_items * 4, experts + pairs / 8, act_rows, s);
    return few_launch<TYPE, 2, true>(a, max_items * 2, experts + pairs / 16, act_rows, s);
}
int launch_gemm_few_grouped(int type, int64_t n, int64_t k, int64_t n_expert, int64_t pairs, int64_t act_rows, const uint8_t *tiles, ActView acts, float *dst, const GroupMap &gm,
                            int64_t max_items, cudaStream_t s) {
    FewArgs a = {};
    for (int e = 0; e < 3; e++) {
        a.tiles[e] = tiles;
        a.dst[e] = dst;
        a.n[e] = a.lddst[e] = n;
        a.tile_start[e] = e ? 0x7fffffff : 0;
    }
    a.tile_start[3] = (int)((n + TILE_ROWS - 1) / TILE_ROWS);
    a.acts = acts;
    a.nb = (int)(k / GROUP_K);
    a.gm = gm;
    a.col_blocks = 1;
    const int rc = device_error_word(&a.err);
    if (rc != B200_STATUS_SUCCESS) return rc;
    switch (type) {
        case B200_TYPE_Q4_K: return few_grouped<B200_TYPE_Q4_K>(a, max_items, n_expert, pairs, act_rows, s);
        case B200_TYPE_Q6_K: return few_grouped<B200_TYPE_Q6_K>(a, max_items, n_expert, pairs, act_rows, s);
        case B200_TYPE_Q8_0: return few_grouped<B200_TYPE_Q8_0>(a, max_items, n_expert, pairs, act_rows, s);
        case B200_TYPE_Q4_0: return few_grouped<B200_TYPE_Q4_0>(a, max_items, n_expert, pairs, act_rows, s);
        case B200_TYPE_MXFP4: return few_grouped<B200_TYPE_MXFP4>(a, max_items, n_expert, pairs, act_rows, s);
        default: B200_REQUIRE(false, "gemm few: no kernel for weight type %d", type);
    }
}

}  // namespace b200
