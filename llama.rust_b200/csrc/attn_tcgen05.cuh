// What the attention kernels on tcgen05 share: barriers, tensor-memory accesses, operand descriptors, pairs of floats.
#pragma once
#include "common.cuh"
#include "tensor_map.h"

namespace b200 {

constexpr uint32_t PA_WAIT_LIMIT = 1u << 20;   // of polls that sleep up to a microsecond each

__device__ __forceinline__ uint32_t pa_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void pa_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(pa_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void pa_arrive(uint64_t *bar) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(pa_smem(bar)) : "memory");
}
__device__ __forceinline__ void pa_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(pa_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool pa_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3; selp.u32 %0, 1, 0, p; }" : "=r"(ok) : "r"(pa_smem(bar)), "r"(parity), "r"(1000u) : "memory");
    return ok != 0;
}
// A warp's: every lane gets the same answer (what follows is done by whole warps).  False: somebody gave up, or this wait did after `limit` polls
__device__ __forceinline__ bool pa_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, uint32_t limit) {
    bool ok = pa_try(bar, parity);
    for (uint32_t it = 1; !ok && it < limit; it++) {
        ok = pa_try(bar, parity);
        if (!ok && (it & 255) == 255 && *abort_flag) break;
    }
    if (__all_sync(0xffffffffu, ok)) return true;
    *abort_flag = 1;
    return false;
}
// what is on its way when a CTA gives up, or ends, is waited for all the same
__device__ __forceinline__ void pa_drain(uint64_t *bar, uint32_t parity, uint32_t limit) {
    for (uint32_t it = 0; it < limit && !pa_try(bar, parity); it++) {}
}
// test hook (b200_debug_attn_wait): polls of a wait, and the visited tile whose values the CTA of the last rows and the first key head does not ask for, -1: none
void attn_wait_hook(uint32_t *limit, int *mute);
__device__ __forceinline__ void pa_tma(uint32_t dst, const CUtensorMap *map, int x, int head, int pos, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(map), "r"(x), "r"(head),
                 "r"(pos), "r"(pa_smem(bar))
                 : "memory");
}
// 128-byte swizzle, 8-row groups 1024 bytes apart; lbo: distance of the 64-element chunks of an MN-major operand
__device__ __forceinline__ uint64_t pa_desc(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void pa_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int acc) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void pa_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, int acc) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void pa_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(pa_smem(bar)) : "memory");
}
__device__ __forceinline__ void pa_ld32(uint32_t *r, uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void pa_st32(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]),
        "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
        "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
        "r"(r[30]), "r"(r[31]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ bool pa_elect() {
    uint32_t ok;
    asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(ok));
    return ok != 0;
}
__device__ __forceinline__ void pa_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void pa_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void pa_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pa_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ float pa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// two floats in one register pair, for the instructions that take two at a time
__device__ __forceinline__ uint64_t pa_pair(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 pa_split(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t pa_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t pa_add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void pa_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t pa_mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float2 pa_ld_peer2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}

// ---- rows whose output is not finite ------------------------------------------------------------------------------
// The products run over whole tiles, so what a cell holds that a row does not see meets that row with weight 0: 0 * Inf and NaN scores spoil it.  A
// row that ends with anything but finite numbers is therefore computed once more, by a warp, from the cells it sees alone: nothing where all is
// finite, and the definition's Inf and NaN where they belong.  (4096 positions take a row about a millisecond; a NaN score, as of a query with a NaN, ends
// it at the first 32: 512 rows of 32 heads over 4096 positions, one query a NaN, 76 us.)
__device__ __forceinline__ bool pa_finite(float x) { return fabsf(x) < INFINITY; }
template <bool BF16>
__device__ __forceinline__ float2 pa_two(uint32_t w) {
    if (BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    return __half22float2(*(const __half2 *)&w);
}
// Row x of the swizzled query operand at q against n entries.  entry(i, &bias, &key, &value): whether the row sees entry i, its addend (log2 units) and
// its 16-byte aligned key and value rows of D elements.  acc[2 e], acc[2 e + 1]: this lane's output channels 64 e + 2 lane and + 1, not yet divided by
// the sum; top: the maximum in use (log2 units, -inf: sees nothing)
template <int D, bool BF16, typename Entry>
__device__ __forceinline__ void pa_row_again(const uint8_t *q, int x, float scale_log2, int n, const Entry &entry, float (&acc)[D / 32], float *top, float *sum) {
    const int lane = threadIdx.x & 31;
    const uint8_t *const qrow = q + (x >> 3) * 1024 + (x & 7) * 128;
    float m = -INFINITY, l = 0.0f;
#pragma unroll
    for (int e = 0; e < D / 32; e++) acc[e] = 0.0f;
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {   // a lane has an entry's score, then two channels of each 64
        const uint8_t *key = nullptr, *value = nullptr;
        float bias = 0.0f, s = -INFINITY;
        const bool sees = base + lane < n && entry(base + lane, &bias, &key, &value);
        if (sees) {
            float dot = 0.0f;
#pragma unroll 2
            for (int c = 0; c < D / 8; c++) {
                const uint4 k4 = *(const uint4 *)(key + 16 * c), q4 = *(const uint4 *)(qrow + (c >> 3) * (128 * 128) + (((c & 7) ^ (x & 7)) << 4));
                const uint32_t kw[4] = {k4.x, k4.y, k4.z, k4.w}, qw[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float2 a = pa_two<BF16>(kw[i]), b = pa_two<BF16>(qw[i]);
                    dot = fmaf(a.x, b.x, dot);
                    dot = fmaf(a.y, b.y, dot);
                }
            }
            s = fmaf(dot, scale_log2, bias);
        }
        if (__any_sync(0xffffffffu, sees && !(s < INFINITY))) {   // NaN, or a weight of exp(inf - inf)
            m = 0.0f;
            l = NAN;
#pragma unroll
            for (int e = 0; e < D / 32; e++) acc[e] = NAN;
            break;
        }
        float mx = s;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (mx == -INFINITY) continue;
        const float mn = fmaxf(m, mx), al = pa_ex2(m - mn), w = pa_ex2(s - mn);
        m = mn;
        float ws = w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ws += __shfl_xor_sync(0xffffffffu, ws, o);
        l = fmaf(l, al, ws);
#pragma unroll
        for (int e = 0; e < D / 32; e++) acc[e] *= al;
        const uint32_t seen = __ballot_sync(0xffffffffu, sees);
#pragma unroll 4
        for (int j = 0; j < 32; j++) {
            const float wj = __shfl_sync(0xffffffffu, w, j);
            const uint8_t *vj = (const uint8_t *)__shfl_sync(0xffffffffu, (unsigned long long)value, j);
            if (!(seen >> j & 1)) continue;
#pragma unroll
            for (int e = 0; e < D / 64; e++) {
                const float2 v = pa_two<BF16>(*(const uint32_t *)(vj + 128 * e + 4 * lane));
                acc[2 * e] = fmaf(wj, v.x, acc[2 * e]);
                acc[2 * e + 1] = fmaf(wj, v.y, acc[2 * e + 1]);
            }
        }
    }
    *top = m;
    *sum = l;
}

}  // namespace b200
