// FLASH_ATTN_EXT, fast mode, prompt batches: attention on the tcgen05 tensor cores, head sizes 64 and 128.
//
//   softmax(q k^T * scale + mask) v        (crates/ggml/src/flash_attn.rs:482-736), for hosts that accept the tolerance asked of
// F16-KV attention (1e-3): q is rounded to f16 as the CPU rounds it (flash_attn.rs:433), the weights of 64 and more query rows are rounded to
// f16 for the second product, those of fewer rows go in as two f16 parts (SPLIT), everything else is F32.
//   * A CTA takes 128 rows of one KV head, a row being (token, query head of the KV head's group) with the heads of a token adjacent,
//     so that every K / V tile and every mask row is shared by the group.  Row r is lane r of tensor memory.
//   * K and V come in tiles of 128 positions by TMA (128-byte swizzle; positions past the cache read as zeros), K a K-major and V an
//     MN-major B operand: a cached row's value elements are contiguous along N, so neither tile is transposed.
//   * (As published with FlashAttention-4:) the tiles that are visited alternate between two groups of four softmax warps.  Each has its own scores (128 columns of
//     tensor memory), its own unnormalised output and its own running maximum and sum, so that one group's exponentials hide the
//     other's products; the two are added at the end.  A thread owns a whole row: no exchange between threads.
//   * The weights go back into tensor memory over the scores they came from, as the A operand of p v: shared memory carries K, V and q only.
//   * With one-part weights the maximum in use is the running one, so that a row's largest weights are exactly 1 and lose nothing.  Let it lag
//     by up to 2^8 and the output is rescaled less often (47 us for the 50 below), but those weights are rounded like any other: 2.05e-4 of
//     float64 for 1.90e-4, and 1.36e-4 for 6.5e-5 with scores three times as wide (maxima per 64 positions, as mma.sync kernels have
//     them: 1.93e-4 and 7.6e-5).  Two parts take no harm from it: there the output is rescaled only when a row's maximum grows by more than
//     2^8 over the one in use, and the sums take the weights as they are.
//   * Two parts cost 14 % at 512 rows over 4096 positions, 8 % at 16 over 2048; 5e-7 to 5e-6 of float64.  The decode kernel, which takes a maximum per
//     16 positions, is 1.4e-4 away (2e-5 with wide scores, 3e-7 where each 16 hold one position that a row sees): one part would be further.
//   * Six warps read the mask ahead of everyone and sort the CTA's (row block, tile) pairs into: all zero (no mask read at all in the
//     softmax), all minus infinity (skipped by every role), mixed (each row reads its 128 mask values).
//   * A row whose output is not finite is computed again from what it sees alone (pa_row_again): the tiles' products multiply hidden cells by 0.
//   * The positions are dealt out to the CTAs of a cluster, tile by tile, where there are too few row blocks for the GPU; the
//     partial outputs meet in shared memory and every CTA finishes its share of the rows.
// Every wait is bounded; a wait that runs out raises the CTA's abort flag and the device error word, and no row of its block is stored.
// What bounds it (512 rows of 32 heads over 4096 positions, 8 KV heads of 128: 50 us; the mma.sync kernel in its place before took 169, 0.19 of
// the rate the products alone would allow): a tile of 128 x 128 costs about 2000 SM clocks, 1024 of them exponentials (16 a clock) and as many
// products, which two groups overlap only in part (tensor pipe busy 30 % of the time, exponentials' pipe 35 %, issue slots 44 %); and about 10 us of a launch are its beginning (q, the first tiles) and end.  On the way: one
// lane that walked the tiles and issued the products with its descriptors in ordinary registers 67.8 us; the warp together, one elected
// lane issuing 57.9; two floats per instruction around the exponentials 53.4; one warp that sorts the tiles for everyone 50.7.
// Not handled here (the caller falls back to the exact kernels): sinks, ALiBi, softcap, dk != dv.
#include <mutex>

#include "attn_tcgen05.cuh"
#include "tensor_map.h"

namespace b200 {

namespace {

constexpr int PA_M = 128, PA_N = 128;                  // rows per CTA, positions per tile
constexpr int PA_MASK_WARPS = 6, PA_SM_WARP0 = 8, PA_THREADS = 512;
constexpr int PA_RING = 16;                            // tiles whose class the mask warps may be ahead
constexpr int PA_MAX_SPLITS = 8;
constexpr int PA_ERR_WAIT = 4;
constexpr float PA_LOG2E = 1.4426950408889634f;
enum { PA_CLEAR = 0, PA_MIXED = 1, PA_HIDDEN = 2 };

template <int D>
struct PaCfg {
    static constexpr int CHUNKS = D / 64;              // 64 elements = one 128-byte swizzled box
    static constexpr int TILE = PA_N * D * 2;
    static constexpr int SLOTS = D == 128 ? 5 : 8;
    static constexpr int PITCH = D + 4;                // floats of a row of the partial output: lanes that own rows fall on different banks
    static constexpr int SMEM = PA_M * D * 2 + SLOTS * TILE + 1024;
    static constexpr uint32_t O_COL = 2 * PA_N;        // tensor memory: two score tiles, then two outputs
    static constexpr uint32_t IDESC_S = (1u << 4) | ((uint32_t)(PA_N >> 3) << 17) | ((uint32_t)(PA_M >> 4) << 24);
    static constexpr uint32_t IDESC_O = (1u << 4) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((uint32_t)(PA_M >> 4) << 24);   // B is MN-major
};
static_assert(PaCfg<128>::SLOTS * PaCfg<128>::TILE >= PA_M * PaCfg<128>::PITCH * 4 && PaCfg<64>::SLOTS * PaCfg<64>::TILE >= PA_M * PaCfg<64>::PITCH * 4, "partial output");

struct PaShared {
    uint64_t empty[8];                     // K / V slots are free
    uint64_t kfirst[2], kv[8];             // K of visited tiles 0 and 1 has landed; V of tile v together with K of tile v + 2
    uint64_t sfull[2], pready[2];          // scores of a group stand; its weights stand
    uint64_t cfull[PA_RING], cempty[PA_RING];
    uint64_t vfull[8], vempty[8];
    uint64_t qready, done;
    int cls[PA_RING];                      // of the CTA's tiles, from the mask warps to the loading one
    int visit[8];                          // the visited tiles: tile * 2 + mixed, -1 behind the last
    int first[2], more[8];                 // whether there is a tile behind kfirst[i]; whether kv[i] has a K
    float ml[2][PA_M][2];                  // maximum and sum of each group's rows, then [0] of the CTA's rows
    uint32_t tmem_base;
    int abort_flag;
};

struct PaArgs {
    const unsigned char *q, *mask, *k, *v;   // k, v: only for rows that are computed again
    int64_t q_nb1, q_nb2, mask_nb1, k_nb1, k_nb2, v_nb1, v_nb2;
    float *dst;
    int64_t n_kv, rows;
    int n_tok, n_head, group, splits, n_tiles, mask_wide;
    float scale_log2, q_sign;
    int *err;
    uint32_t wait_limit;
    int mute;   // test hook
};

template <int D, bool SPLIT>
__global__ void __launch_bounds__(PA_THREADS, 1)
fa_prompt_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, const PaArgs a) {
    using C = PaCfg<D>;
    constexpr float LAZY = SPLIT ? 8.0f : 0.0f;   // log2 of the growth of a maximum that is let pass
    extern __shared__ uint8_t pa_raw[];
    __shared__ PaShared sh;
    pdl_trigger();
    const uint32_t q_s = (pa_smem(pa_raw) + 1023u) & ~1023u, kv_s = q_s + PA_M * D * 2;
    uint8_t *const q_g = pa_raw + (q_s - pa_smem(pa_raw));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    volatile int *abort_flag = &sh.abort_flag;
    const int rank = (int)(blockIdx.x % (unsigned)a.splits), hk = blockIdx.y;
    // the last row blocks of a causal prompt see most: they start first
    const int64_t row0 = ((int64_t)gridDim.x / a.splits - 1 - (int64_t)(blockIdx.x / (unsigned)a.splits)) * PA_M;
    const int tok0 = (int)(row0 / a.group);
    const int64_t row_last = row0 + PA_M - 1 < a.rows - 1 ? row0 + PA_M - 1 : a.rows - 1;
    const int n_tok_blk = (int)(row_last / a.group) - tok0 + 1;
    const int n_mine = rank < a.n_tiles ? (a.n_tiles - 1 - rank) / a.splits + 1 : 0;   // tiles rank, rank + splits, ..
    const bool ragged = a.n_kv % PA_N != 0;

    if (tid == 0) {
        for (int i = 0; i < 8; i++) {
            pa_init(&sh.empty[i], 1);
            pa_init(&sh.vfull[i], 1);
            pa_init(&sh.vempty[i], 4);
            pa_init(&sh.kv[i], 1);
        }
        for (int g = 0; g < 2; g++) {
            pa_init(&sh.kfirst[g], 1);
            pa_init(&sh.sfull[g], 1);
            pa_init(&sh.pready[g], 4);
        }
        for (int i = 0; i < PA_RING; i++) {
            pa_init(&sh.cfull[i], 1);
            pa_init(&sh.cempty[i], 1);
        }
        pa_init(&sh.qready, 8);
        pa_init(&sh.done, 1);
        sh.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        // all 512 columns: the operand slots fill the SM's shared memory, so no second CTA competes for them
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pa_smem(&sh.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pa_fence_before();
    __syncthreads();
    pa_fence_after();
    const uint32_t tmem = sh.tmem_base;
    pdl_wait();   // q, the cache rows of this step and the mask come from earlier kernels / copies

    if (warp < PA_SM_WARP0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == 0) {
            // walks the tiles, sorts out the hidden ones, tells the softmax groups which tiles are theirs (visited tile v: group v % 2) and loads:
            // K 0, K 1, then V v and K v + 2, the order in which the products read them
            int seq = 0, i = 0, v_told = 0;
            // the next visited tile as the softmax groups get it; -1: none (or winding down)
            auto next_visit = [&]() -> int {
                while (i < n_mine) {
                    const int tile = rank + i * a.splits, s = i % PA_RING;
                    int c = ragged && tile == a.n_tiles - 1 ? PA_MIXED : PA_CLEAR;
                    if (a.mask) {
                        if (!pa_wait(&sh.cfull[s], (uint32_t)(i / PA_RING) & 1u, abort_flag, a.wait_limit)) break;
                        c = *(volatile int *)&sh.cls[s];
                        __syncwarp();
                        if (lane == 0) pa_arrive(&sh.cempty[s]);
                    }
                    i++;
                    if (c != PA_HIDDEN) return tile * 2 + (c == PA_MIXED);
                }
                i = n_mine;
                return -1;
            };
            auto tell = [&](int t) {
                const int s = v_told % 8;
                if (v_told >= 8 && !pa_wait(&sh.vempty[s], ((uint32_t)(v_told / 8) & 1u) ^ 1u, abort_flag, a.wait_limit)) return false;
                if (lane == 0) {
                    *(volatile int *)&sh.visit[s] = t;
                    pa_arrive(&sh.vfull[s]);
                }
                v_told++;
                return true;
            };
            auto wait_slot = [&]() { return pa_wait(&sh.empty[seq % C::SLOTS], ((uint32_t)(seq / C::SLOTS) & 1u) ^ 1u, abort_flag, a.wait_limit); };
            auto load = [&](const CUtensorMap *map, int t, uint64_t *bar) {   // into slot `seq`, by lane 0
                if (lane == 0) {
#pragma unroll
                    for (int c = 0; c < C::CHUNKS; c++) pa_tma(kv_s + (uint32_t)((seq % C::SLOTS) * C::TILE + c * PA_N * 128), map, 64 * c, hk, (t >> 1) * PA_N, bar);
                }
                seq++;
            };
            const int mute = (blockIdx.x | blockIdx.y) == 0 ? a.mute : -1;
            bool ok = true;
            int t[2];
            for (int g = 0; g < 2; g++) {
                t[g] = next_visit();
                ok = ok && tell(t[g]);
                if (lane == 0) {
                    *(volatile int *)&sh.first[g] = t[g] >= 0;
                    if (t[g] >= 0) pa_expect(&sh.kfirst[g], C::TILE);
                    else pa_arrive(&sh.kfirst[g]);
                }
                if (t[g] >= 0) load(&kmap, t[g], &sh.kfirst[g]);   // the slots are free
            }
            int v = 0, begun = 0;   // copies of kv phases 0 .. begun - 1 were started.  A slot of V is waited for that belonged to a tile at most six
                                // before: phase v - 8 is long through
            while (ok && t[0] >= 0) {
                const int cur = t[0];
                t[0] = t[1];
                t[1] = next_visit();
                ok = tell(t[1]) && wait_slot();   // in the end both groups have been told that there is no more
                if (!ok) break;
                const bool more = t[1] >= 0;
                if (lane == 0) {
                    *(volatile int *)&sh.more[v % 8] = more;
                    pa_expect(&sh.kv[v % 8], more ? 2 * C::TILE : C::TILE);
                }
                if (v != mute) load(&vmap, cur, &sh.kv[v % 8]);
                else seq++;
                begun = v + 1;
                if (more) {
                    ok = wait_slot();
                    if (!ok && lane == 0) asm volatile("mbarrier.complete_tx.shared::cta.relaxed.cta.b64 [%0], %1;" ::"r"(pa_smem(&sh.kv[v % 8])), "r"(C::TILE) : "memory");
                    if (ok) load(&kmap, t[1], &sh.kv[v % 8]);
                }
                v++;
            }
            // a CTA that gives up still waits (bounded) for the copies it has in flight
            if (*abort_flag) {
                for (int g = 0; g < 2; g++) pa_drain(&sh.kfirst[g], 0, a.wait_limit);
                for (int p = begun > 8 ? begun - 8 : 0; p < begun; p++) pa_drain(&sh.kv[p % 8], (uint32_t)(p / 8) & 1u, a.wait_limit);
            }
        } else if (warp == 1) {
            // the whole warp waits, one elected lane issues: descriptors then stay in uniform registers
            const bool leader = pa_elect();
            int seq = 0, scored = 0;
            const uint64_t q_desc = pa_desc(q_s, 16), k_desc = pa_desc(kv_s, 16), v_desc = pa_desc(kv_s, PA_N * 128);
            // scores of the tile in slot `seq`, for group g: over its former weights, whose product was issued before (products complete in order)
            auto scores = [&](int g) {
                const int s = seq % C::SLOTS;
                if (leader) {
#pragma unroll
                    for (int ks = 0; ks < D / 16; ks++) {
                        const uint32_t off = (uint32_t)((ks >> 2) * PA_M * 128 + (ks & 3) * 32) >> 4;
                        pa_mma_ss(tmem + (uint32_t)(g * PA_N), q_desc + off, k_desc + (uint32_t)(s * (C::TILE >> 4)) + off, C::IDESC_S, ks > 0);
                    }
                    pa_commit(&sh.empty[s]);
                    pa_commit(&sh.sfull[g]);
                }
                seq++;
                scored++;
            };
            bool ok = pa_wait(&sh.qready, 0, abort_flag, a.wait_limit);
            for (int g = 0; g < 2 && ok; g++) {
                ok = pa_wait(&sh.kfirst[g], 0, abort_flag, a.wait_limit);
                pa_fence_after();
                if (ok && *(volatile int *)&sh.first[g]) scores(g);
            }
            for (int v = 0; v < scored && ok; v++) {
                const int g = v & 1, j = v >> 1, s = seq % C::SLOTS;
                // what the products read, then the weights: from there on nothing is waited for
                ok = pa_wait(&sh.kv[v % 8], (uint32_t)(v / 8) & 1u, abort_flag, a.wait_limit);
                const bool more = *(volatile int *)&sh.more[v % 8];
                ok = ok && pa_wait(&sh.pready[g], (uint32_t)j & 1u, abort_flag, a.wait_limit);
                if (!ok) break;
                pa_fence_after();
                if (leader) {
#pragma unroll
                    for (int part = 0; part < (SPLIT ? 2 : 1); part++)   // the weights' high parts, then their low parts
#pragma unroll
                        for (int ks = 0; ks < PA_N / 16; ks++)
                            pa_mma_ts(tmem + C::O_COL + (uint32_t)(g * D), tmem + (uint32_t)(g * PA_N + part * 64 + ks * 8), v_desc + (uint32_t)(s * (C::TILE >> 4) + ks * 128),
                                      C::IDESC_O, j > 0 || ks > 0 || part > 0);
                    pa_commit(&sh.empty[s]);
                }
                seq++;
                if (more) scores(g);
            }
            if (leader) pa_commit(&sh.done);
            // the operands and tensor memory stay until the products are through, whatever the other roles do
            pa_drain(&sh.done, 0, a.wait_limit);
        } else if (a.mask) {
            // 16-byte pieces on their boundaries, 16 of a token's 256 bytes and a 17th where they do not begin on one.  What such a piece shares
            // with its neighbours is counted too: a tile then is at worst mixed where it could have been clear or hidden
            const uintptr_t m_lo = (uintptr_t)a.mask, m_hi = m_lo + (uintptr_t)(a.n_tok - 1) * a.mask_nb1 + (uintptr_t)a.n_kv * 2;
            const uint32_t hidden2 = 0xFC00FC00u;
            for (int i = warp - 2; i < n_mine; i += PA_MASK_WARPS) {
                const int tile = rank + i * a.splits, s = i % PA_RING;
                const uintptr_t src = m_lo + (uintptr_t)tok0 * a.mask_nb1 + (uintptr_t)tile * (PA_N * 2);
                const int64_t left = a.n_kv - (int64_t)tile * PA_N;
                const int bytes = left < PA_N ? (int)left * 2 : PA_N * 2;
                uint32_t any = bytes < PA_N * 2;   // some value is not zero
                uint32_t seen = 0;                 // some value is not minus infinity
                auto piece = [&](uintptr_t row, int c) -> uint4 {
                    const uintptr_t at = (row & ~(uintptr_t)15) + (uintptr_t)c;
                    uint4 v = make_uint4(0, 0, 0, 0);
                    if (at >= row + (uintptr_t)bytes) return make_uint4(hidden2, hidden2, hidden2, hidden2);   // past the row: only where any is set
                    if (at >= m_lo && at + 16 <= m_hi) return *(const uint4 *)at;
                    uint32_t h[8];   // the ends of the mask's memory
#pragma unroll
                    for (int e = 0; e < 8; e++) h[e] = at + 2 * e >= m_lo && at + 2 * e < m_hi ? *(const uint16_t *)(at + 2 * e) : 0xFC00u;
                    any |= 1;
                    v.x = h[0] | h[1] << 16;
                    v.y = h[2] | h[3] << 16;
                    v.z = h[4] | h[5] << 16;
                    v.w = h[6] | h[7] << 16;
                    return v;
                };
                auto count = [&](const uint4 &v) {
                    any |= v.x | v.y | v.z | v.w;
                    seen |= (v.x ^ hidden2) | (v.y ^ hidden2) | (v.z ^ hidden2) | (v.w ^ hidden2);
                };
                const int half = lane >> 4, c = (lane & 15) * 16;
                if (a.mask_wide && bytes == PA_N * 2) {
                    const unsigned char *p = (const unsigned char *)src + half * a.mask_nb1 + c;
                    for (int t = half; t < n_tok_blk; t += 16, p += 16 * a.mask_nb1) {
                        uint4 v[8];
#pragma unroll
                        for (int u = 0; u < 8; u++) v[u] = *(const uint4 *)(t + 2 * u < n_tok_blk ? p + 2 * u * a.mask_nb1 : p);
#pragma unroll
                        for (int u = 0; u < 8; u++) count(v[u]);
                    }
                } else {
                    for (int t = half; t < n_tok_blk; t += 8) {
                        uint4 v[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) v[u] = piece(src + (uintptr_t)(t + 2 * u < n_tok_blk ? t + 2 * u : t) * a.mask_nb1, c);
#pragma unroll
                        for (int u = 0; u < 4; u++) count(v[u]);
                    }
                    if (!a.mask_wide)
                        for (int t = lane; t < n_tok_blk; t += 32) {
                            const uintptr_t row = src + (uintptr_t)t * a.mask_nb1;
                            if (row & 15) count(piece(row, 256));
                        }
                }
                const bool w_any = __any_sync(0xffffffffu, any != 0), w_seen = __any_sync(0xffffffffu, seen != 0);
                if (i >= PA_RING && !pa_wait(&sh.cempty[s], ((uint32_t)(i / PA_RING) & 1u) ^ 1u, abort_flag, a.wait_limit)) break;
                if (lane == 0) {
                    *(volatile int *)&sh.cls[s] = !w_seen ? PA_HIDDEN : w_any ? PA_MIXED : PA_CLEAR;
                    pa_arrive(&sh.cfull[s]);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
        const int g = (warp - PA_SM_WARP0) >> 2, r = (warp & 3) * 32 + lane;   // group, row: a warp reaches the tensor-memory lanes of its number modulo 4
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t t_s = tmem + lanes + (uint32_t)(g * PA_N), t_o = tmem + lanes + C::O_COL + (uint32_t)(g * D);
        const int64_t row = row0 + r;
        const bool live = row < a.rows;
        const int tok = live ? (int)(row / a.group) : tok0;
        {
            // q as f16 into the swizzled K-major operand: a warp takes 16 rows, lane = two neighbouring elements of each 64 (a thread per row would
            // touch 32 lines with every load: 128 rows took 9 us that way, 1.5 like this)
            constexpr int RW = 16;
            const int rw0 = (warp - PA_SM_WARP0) * RW;
#pragma unroll
            for (int h = 0; h < RW; h += 8) {
                float2 f[8][C::CHUNKS];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int64_t rr = row0 + rw0 + h + u;
                    const int tk = (int)(rr / a.group), hd = hk * a.group + (int)(rr - (int64_t)tk * a.group);
                    const float *src = (const float *)(a.q + (int64_t)tk * a.q_nb1 + (int64_t)hd * a.q_nb2) + 2 * lane;
#pragma unroll
                    for (int c = 0; c < C::CHUNKS; c++) f[u][c] = rr < a.rows ? *(const float2 *)(src + 64 * c) : make_float2(0.0f, 0.0f);
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int x = rw0 + h + u;
#pragma unroll
                    for (int c = 0; c < C::CHUNKS; c++) {
                        const __half2 w = __floats2half2_rn(f[u][c].x * a.q_sign, f[u][c].y * a.q_sign);
                        *(__half2 *)(q_g + c * (PA_M * 128) + (x >> 3) * 1024 + (x & 7) * 128 + ((((lane >> 2) ^ (x & 7)) << 4) | (lane & 3) * 4)) = w;
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) pa_arrive(&sh.qready);
        }
        float m = -INFINITY, l = 0.0f;   // the maximum in use (log2 units) and the sum of the weights under it
        const unsigned char *mrow = a.mask ? a.mask + (int64_t)tok * a.mask_nb1 : nullptr;
        for (int j = 0;; j++) {
            const int v = 2 * j + g;
            if (!pa_wait(&sh.vfull[v % 8], (uint32_t)(v / 8) & 1u, abort_flag, a.wait_limit)) break;
            const int visit = *(volatile int *)&sh.visit[v % 8];
            __syncwarp();
            if (lane == 0) pa_arrive(&sh.vempty[v % 8]);
            if (visit < 0) break;
            const bool mixed = visit & 1;
            const int64_t pos0 = (int64_t)(visit >> 1) * PA_N;
            uint32_t s[PA_N];
            float sc = a.scale_log2;
            if (!mixed) {
                if (!pa_wait(&sh.sfull[g], (uint32_t)j & 1u, abort_flag, a.wait_limit)) break;
                pa_fence_after();
#pragma unroll
                for (int c = 0; c < PA_N; c += 32) pa_ld32(s + c, t_s + (uint32_t)c);
                pa_wait_ld();
            } else {
                // the row's mask values while the scores are computed
                uint32_t w[PA_N / 2];
#pragma unroll
                for (int c = 0; c < PA_N; c += 32) {
                    const unsigned char *at = mrow + (pos0 + c) * 2;
                    uint32_t *wc = w + c / 2;
                    if (pos0 + c + 32 > a.n_kv || !mrow) {
#pragma unroll
                        for (int e = 0; e < 16; e++) {
                            const int64_t p = pos0 + c + 2 * e;
                            const uint32_t lo = p >= a.n_kv ? 0xFC00u : mrow ? *(const uint16_t *)(at + 4 * e) : 0u;
                            const uint32_t hi = p + 1 >= a.n_kv ? 0xFC00u : mrow ? *(const uint16_t *)(at + 4 * e + 2) : 0u;
                            wc[e] = lo | hi << 16;
                        }
                    } else if (a.mask_wide) {
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const uint4 x = *(const uint4 *)(at + e * 16);
                            wc[4 * e] = x.x;
                            wc[4 * e + 1] = x.y;
                            wc[4 * e + 2] = x.z;
                            wc[4 * e + 3] = x.w;
                        }
                    } else if (((uintptr_t)at & 2) == 0) {
#pragma unroll
                        for (int e = 0; e < 16; e++) wc[e] = *(const uint32_t *)(at + 4 * e);
                    } else {   // a row that starts between two words: a half, 15 words, a half
                        uint32_t before = (uint32_t)*(const uint16_t *)at << 16;
#pragma unroll
                        for (int e = 0; e < 16; e++) {
                            const uint32_t next = e < 15 ? *(const uint32_t *)(at + 4 * e + 2) : (uint32_t)*(const uint16_t *)(at + 62);
                            wc[e] = before >> 16 | next << 16;
                            before = next;
                        }
                    }
                }
                if (!pa_wait(&sh.sfull[g], (uint32_t)j & 1u, abort_flag, a.wait_limit)) break;
                pa_fence_after();
                sc = 1.0f;
#pragma unroll
                for (int c = 0; c < PA_N; c += 32) {
                    pa_ld32(s + c, t_s + (uint32_t)c);
                    pa_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; e++) {
                        const float2 f = __half22float2(*(const __half2 *)&w[c / 2 + e]);
                        s[c + 2 * e] = __float_as_uint(fmaf(__uint_as_float(s[c + 2 * e]), a.scale_log2, f.x * PA_LOG2E));
                        s[c + 2 * e + 1] = __float_as_uint(fmaf(__uint_as_float(s[c + 2 * e + 1]), a.scale_log2, f.y * PA_LOG2E));
                    }
                }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < PA_N; c += 8)
#pragma unroll
                for (int e = 0; e < 4; e++) mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(s[c + e]), __uint_as_float(s[c + 4 + e])));
            const float top = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc);
            if (j == 0) {
                m = top;
            } else {
                const bool grow = top > m + LAZY;   // also when nothing was seen before
                if (__any_sync(0xffffffffu, grow)) {
                    // the group's former product is complete: the scores that were waited for were issued behind it
                    const float al = grow ? pa_ex2(m - top) : 1.0f;
                    if (grow) m = top;
                    l *= al;
#pragma unroll 1
                    for (int c = 0; c < D; c += 32) {
                        uint32_t o[32];
                        pa_ld32(o, t_o + (uint32_t)c);
                        pa_wait_ld();
#pragma unroll
                        for (int e = 0; e < 32; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * al);
                        pa_st32(t_o + (uint32_t)c, o);
                    }
                    pa_wait_st();
                }
            }
            const float sub = m == -INFINITY ? 0.0f : m;   // a row that sees nothing yet: weights of zero
            uint64_t ps[2] = {0, 0};   // two running sums each
            const uint64_t sc2 = pa_pair(sc, sc), sub2 = pa_pair(-sub, -sub);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t p[32], low[SPLIT ? 32 : 1];
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    const float2 x = pa_split(pa_fma2(pa_pair(__uint_as_float(s[64 * h + 2 * c]), __uint_as_float(s[64 * h + 2 * c + 1])), sc2, sub2));
                    const float2 e = make_float2(pa_ex2(x.x), pa_ex2(x.y));
                    const __half2 w = __floats2half2_rn(e.x, e.y);
                    const float2 f = __half22float2(w);
                    p[c] = *(const uint32_t *)&w;
                    if (SPLIT) {
                        const __half2 rest = __floats2half2_rn(e.x - f.x, e.y - f.y);
                        low[SPLIT ? c : 0] = *(const uint32_t *)&rest;
                        ps[c & 1] = pa_add2(ps[c & 1], pa_pair(e.x, e.y));
                    } else {
                        // the sum takes the weights as the second product will see them (rounded to f16): what is common to a row's
                        // numerator and denominator cancels
                        ps[c & 1] = pa_add2(ps[c & 1], pa_pair(f.x, f.y));
                    }
                }
                pa_st32(t_s + (uint32_t)(32 * h), p);
                if (SPLIT) pa_st32(t_s + (uint32_t)(64 + 32 * h), low);
            }
            const float2 p0 = pa_split(ps[0]), p1 = pa_split(ps[1]);
            l += (p0.x + p1.x) + (p0.y + p1.y);
            pa_wait_st();
            pa_fence_before();
            __syncwarp();
            if (lane == 0) pa_arrive(&sh.pready[g]);
        }
        sh.ml[g][r][0] = m;
        sh.ml[g][r][1] = l;
        const bool finished = __all_sync(0xffffffffu, pa_wait(&sh.done, 0, abort_flag, a.wait_limit) && !*abort_flag);
        pa_fence_after();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const float ma = sh.ml[0][r][0], mb = sh.ml[1][r][0], mm = fmaxf(ma, mb);
        // No output where the group visited no tile or the row saw nothing in them.  Their sum is 0 then, or NaN: a maximum does not show a NaN
        const bool ina = ma != -INFINITY, inb = mb != -INFINITY;
        const float wa = ina ? pa_ex2(ma - mm) : 1.0f, wb = inb ? pa_ex2(mb - mm) : 1.0f;
        const float lt = wa * sh.ml[0][r][1] + wb * sh.ml[1][r][1];
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (g == 0) {
            sh.ml[0][r][0] = mm;
            sh.ml[0][r][1] = lt;
        }
        if (finished) {
            float *part = (float *)(q_g + PA_M * D * 2) + (size_t)r * C::PITCH;   // over the K / V slots
#pragma unroll 1
            for (int c = g * (D / 2); c < (g + 1) * (D / 2); c += 32) {
                uint32_t x[32], y[32];
                pa_ld32(x, tmem + lanes + C::O_COL + (uint32_t)c);
                pa_ld32(y, tmem + lanes + C::O_COL + (uint32_t)(D + c));
                pa_wait_ld();
#pragma unroll
                for (int e = 0; e < 32; e++) {
                    const float u = ina ? wa * __uint_as_float(x[e]) : 0.0f, v = inb ? wb * __uint_as_float(y[e]) : 0.0f;
                    x[e] = __float_as_uint(u + v);
                }
#pragma unroll
                for (int e = 0; e < 32; e += 4) *(uint4 *)(part + c + e) = make_uint4(x[e], x[e + 1], x[e + 2], x[e + 3]);
            }
        }
        pa_fence_before();
    }
    __syncthreads();
    pa_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    if (*abort_flag) {   // no row of this block is stored, by whichever CTA of the cluster: a maximum of NaN, which no row has otherwise, says so
        if (tid == 0) atomicExch(a.err, PA_ERR_WAIT);
        if (tid < PA_M) sh.ml[0][tid][0] = NAN;
        __syncthreads();
    }
    if (a.splits > 1) pa_cluster_sync();
    {
        // this CTA's share of the rows: a warp per row, the CTAs' partial outputs under their common maximum
        const int lo = PA_M * rank / a.splits, hi = PA_M * (rank + 1) / a.splits;
        const uint32_t ml = pa_smem(&sh.ml[0][0][0]);
        uint32_t again = 0;   // which of this warp's rows are not finite
        for (int r = lo + warp; r < hi; r += PA_THREADS / 32) {
            const int64_t row = row0 + r;
            if (row >= a.rows) break;
            float2 st[PA_MAX_SPLITS];
            float top = -INFINITY;
            bool whole = true;
#pragma unroll
            for (int p = 0; p < PA_MAX_SPLITS; p++) {
                st[p] = p < a.splits ? pa_ld_peer2(pa_mapa(ml + (uint32_t)r * 8, (uint32_t)p)) : make_float2(-INFINITY, 0.0f);
                top = fmaxf(top, st[p].x);
                whole = whole && st[p].x == st[p].x;
            }
            if (!whole) continue;
            float sum = 0.0f, acc[D / 32];
#pragma unroll
            for (int e = 0; e < D / 32; e++) acc[e] = 0.0f;
#pragma unroll
            for (int p = 0; p < PA_MAX_SPLITS; p++) {
                if (st[p].x == -INFINITY) {
                    sum += st[p].y;   // 0 or NaN
                    continue;
                }
                const float w = pa_ex2(st[p].x - top);
                sum += w * st[p].y;
                const uint32_t src = pa_mapa(kv_s + (uint32_t)(r * C::PITCH + lane * 2) * 4, (uint32_t)p);
#pragma unroll
                for (int e = 0; e < D / 64; e++) {
                    const float2 v = pa_ld_peer2(src + (uint32_t)e * 256);
                    acc[2 * e] += w * v.x;
                    acc[2 * e + 1] += w * v.y;
                }
            }
            bool fine = pa_finite(sum);
#pragma unroll
            for (int e = 0; e < D / 32; e++) fine = fine && pa_finite(acc[e]);
            if (!__all_sync(0xffffffffu, fine)) again |= 1u << ((r - lo - warp) / (PA_THREADS / 32));
            const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;   // a row that sees nothing gives zeros, as on the CPU
            const int tok = (int)(row / a.group), head = hk * a.group + (int)(row - (int64_t)tok * a.group);
            float *out = a.dst + ((int64_t)tok * a.n_head + head) * D + lane * 2;
#pragma unroll
            for (int e = 0; e < D / 64; e++) *(float2 *)(out + e * 64) = make_float2(acc[2 * e] * inv, acc[2 * e + 1] * inv);
        }
#pragma unroll 1
        for (; again; again &= again - 1) {
            const int r = lo + warp + (__ffs(again) - 1) * (PA_THREADS / 32);
            const int64_t row = row0 + r;
            const int tok = (int)(row / a.group), head = hk * a.group + (int)(row - (int64_t)tok * a.group);
            const uint8_t *const k = a.k + (int64_t)hk * a.k_nb2, *const v = a.v + (int64_t)hk * a.v_nb2;
            const uint16_t *const seen = a.mask ? (const uint16_t *)(a.mask + (int64_t)tok * a.mask_nb1) : nullptr;
            float acc[D / 32], top, sum;
            pa_row_again<D, false>(q_g, r, a.scale_log2, (int)a.n_kv, [&](int i, float *bias, const uint8_t **key, const uint8_t **value) {
                if (seen) {
                    if (seen[i] == 0xFC00) return false;
                    *bias = f16_bits_to_f32(seen[i]) * PA_LOG2E;
                }
                *key = k + i * a.k_nb1;
                *value = v + i * a.v_nb1;
                return true;
            }, acc, &top, &sum);
            const float inv = sum == 0.0f ? 0.0f : 1.0f / sum;
            float *out = a.dst + ((int64_t)tok * a.n_head + head) * D + lane * 2;
#pragma unroll
            for (int e = 0; e < D / 64; e++) *(float2 *)(out + e * 64) = make_float2(acc[2 * e] * inv, acc[2 * e + 1] * inv);
        }
    }
    if (a.splits > 1) pa_cluster_sync();   // nobody's shared memory goes while a peer reads it
}

// CTAs of a cluster that share the positions of a row block: the number that takes the fewest tile steps in all waves, given how many clusters
// of each size the GPU runs at once (clusters[s - 1]; its partitions differ in size, so it is asked).  A wave costs about four tile steps
// besides its tiles (q, the first tiles, the merge).
int pick_splits(int64_t blocks, int64_t tiles, const int *clusters) {
    int best = 1;
    int64_t cost = INT64_MAX;
    for (int s = 1; s <= PA_MAX_SPLITS && s <= tiles; s++) {
        if (clusters[s - 1] < 1) continue;
        const int64_t c = ((blocks + clusters[s - 1] - 1) / clusters[s - 1]) * ((tiles + s - 1) / s + 4 + (s > 1));
        if (c < cost) {
            cost = c;
            best = s;
        }
    }
    return best;
}

// the [n_kv][n_head_kv][D] f16 view as boxes of 64 elements x 128 positions of one head
bool cache_map(CUtensorMap *map, const void *base, int D, int64_t heads, int64_t n_kv, int64_t nb1, int64_t nb2) {
    if (heads == 1) nb2 = (int64_t)D * 2;
    if (n_kv == 1) nb1 = (int64_t)D * 2;
    return cache_tile_map(map, base, D, heads, n_kv, nb1, nb2, PA_N);
}

template <int D, bool SPLIT>
int launch(const CUtensorMap &km, const CUtensorMap &vm, PaArgs &p, int64_t blocks, int64_t heads, int dev, cudaStream_t s) {
    static std::mutex mu;
    static int clusters[64][PA_MAX_SPLITS];
    static bool known[64] = {};
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!known[dev]) {
            B200_CUDA(cudaFuncSetAttribute(fa_prompt_kernel<D, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, PaCfg<D>::SMEM));
            B200_CUDA(cudaDeviceGetAttribute(&clusters[dev][0], cudaDevAttrMultiProcessorCount, dev));
            for (int n = 2; n <= PA_MAX_SPLITS; n++) {
                cudaLaunchConfig_t cfg = {};
                cudaLaunchAttribute attr[1];
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = n;
                attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
                cfg.gridDim = dim3(n);
                cfg.blockDim = dim3(PA_THREADS);
                cfg.dynamicSmemBytes = PaCfg<D>::SMEM;
                cfg.attrs = attr;
                cfg.numAttrs = 1;
                if (cudaOccupancyMaxActiveClusters(&clusters[dev][n - 1], fa_prompt_kernel<D, SPLIT>, &cfg) != cudaSuccess) {
                    cudaGetLastError();
                    clusters[dev][n - 1] = 0;
                }
            }
            known[dev] = true;
        }
    }
    p.splits = pick_splits(blocks * heads, p.n_tiles, clusters[dev]);
    const dim3 grid((unsigned)(blocks * p.splits), (unsigned)heads);
    if (p.splits == 1) return launch_pdl(fa_prompt_kernel<D, SPLIT>, grid, dim3(PA_THREADS), PaCfg<D>::SMEM, s, km, vm, p);
    return launch_pdl_cluster(fa_prompt_kernel<D, SPLIT>, grid, dim3(PA_THREADS), (unsigned)p.splits, PaCfg<D>::SMEM, s, km, vm, p);
}

uint32_t g_attn_wait_limit = 0;
int g_attn_mute = -1;

}  // namespace

void attn_debug_wait(int spin_limit, int mute_tile) {
    g_attn_wait_limit = spin_limit > 0 ? (uint32_t)spin_limit : 0u;
    g_attn_mute = mute_tile;
}
void attn_wait_hook(uint32_t *limit, int *mute) {
    *limit = g_attn_wait_limit ? g_attn_wait_limit : PA_WAIT_LIMIT;
    *mute = g_attn_wait_limit ? g_attn_mute : -1;
}

// true: the fast prompt kernel took the call (*rc is its status); false: not a shape it handles.  Which of 2 to 63 rows come here: flash_attn.cu
bool flash_attn_fast_prompt(const b200_flash_attn_args *a, cudaStream_t s, int *rc) {
    *rc = B200_STATUS_SUCCESS;
    if (a->sinks || a->max_bias != 0.0f || a->logit_softcap != 0.0f || a->dk != a->dv || (a->dk != 64 && a->dk != 128) || a->n_kv == 0 || a->n_tok == 0)
        return false;
    if (a->q_nb1 % 8 || a->q_nb2 % 8 || ((uintptr_t)a->q & 7) || ((uintptr_t)a->dst & 7) || a->n_head % a->n_head_kv) return false;
    if (a->k_nb1 % 16 || a->v_nb1 % 16 || a->k_nb2 % 16 || a->v_nb2 % 16 || ((uintptr_t)a->k & 15) || ((uintptr_t)a->v & 15)) return false;
    if (a->mask && (a->mask_nb1 % 2 || ((uintptr_t)a->mask & 1))) return false;
    const int64_t group = a->n_head / a->n_head_kv, rows = a->n_tok * group, blocks = (rows + PA_M - 1) / PA_M, tiles = (a->n_kv + PA_N - 1) / PA_N;
    if (a->n_tok > 0x7fffffffLL || blocks * PA_MAX_SPLITS > 0x7fffffffLL || a->n_head_kv > 65535 || a->n_kv > 0x7fffff00LL) return false;
    const int D = (int)a->dk;
    PaArgs p;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) {
        *rc = cuda_fail(e, "flash_attn prompt: device query", __FILE__, __LINE__);
        return true;
    }
    CUtensorMap km, vm;
    if (!cache_map(&km, a->k, D, a->n_head_kv, a->n_kv, a->k_nb1, a->k_nb2) || !cache_map(&vm, a->v, D, a->n_head_kv, a->n_kv, a->v_nb1, a->v_nb2)) return false;
    *rc = device_error_word(&p.err);
    if (*rc != B200_STATUS_SUCCESS) return true;
    p.q = (const unsigned char *)a->q;
    p.q_nb1 = a->q_nb1;
    p.q_nb2 = a->q_nb2;
    p.mask = (const unsigned char *)a->mask;
    p.mask_nb1 = a->mask_nb1;
    p.mask_wide = a->mask && a->mask_nb1 % 16 == 0 && ((uintptr_t)a->mask & 15) == 0;
    p.k = (const unsigned char *)a->k;
    p.v = (const unsigned char *)a->v;
    p.k_nb1 = a->k_nb1;
    p.k_nb2 = a->k_nb2;
    p.v_nb1 = a->v_nb1;
    p.v_nb2 = a->v_nb2;
    attn_wait_hook(&p.wait_limit, &p.mute);
    p.dst = a->dst;
    p.n_kv = a->n_kv;
    p.rows = rows;
    p.n_tok = (int)a->n_tok;
    p.n_head = (int)a->n_head;
    p.group = (int)group;
    p.n_tiles = (int)tiles;
    // a row's maximum is taken before the scale, which must then not be negative: its sign goes to q
    p.scale_log2 = fabsf(a->scale) * PA_LOG2E;
    p.q_sign = a->scale < 0.0f ? -1.0f : 1.0f;
    // two-part weights where the decode kernel's are the measure
    if (a->n_tok < 64) *rc = D == 128 ? launch<128, true>(km, vm, p, blocks, a->n_head_kv, dev, s) : launch<64, true>(km, vm, p, blocks, a->n_head_kv, dev, s);
    else *rc = D == 128 ? launch<128, false>(km, vm, p, blocks, a->n_head_kv, dev, s) : launch<64, false>(km, vm, p, blocks, a->n_head_kv, dev, s);
    return true;
}

}  // namespace b200
