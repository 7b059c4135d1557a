// Grouped-query attention of a prompt's rows over BF16 cells on the tcgen05 tensor cores: the function of grouped_attn_mma_kernel
// (grouped_attn.cu: window, kept first positions, sinks, rotated queries, entries that lead to cells), for keys and values of 64 or 128 channels (D) and
// key heads that a power of two of query heads shares.
//
// The frame is fa_prompt_kernel's (flash_attn_prompt.cu): 128 rows of one key head, a row being (token, query head), two groups of four softmax
// warps that take turns at tiles of 128 entries, scores, weights and unnormalised outputs in tensor memory, a rescaling of the output only
// when a maximum grows by more than 2^8.  What differs:
//   * an entry's cell can be anywhere.  A lane of the loading warp looks up the cells of four entries, two tiles ahead; 32 entries whose cells stand
//     one after the other (a prompt's mostly do) come by one tensor-map copy of 32 rows, others by gathering copies of four rows each;
//   * a weight stays a 32-bit value to 2^-17: it enters the second product as two BF16 parts, each half of the tensor-memory columns its score
//     came from, with two sets of MMAs;
//   * a row whose output is not finite is computed again from the entries it sees alone (pa_row_again): the products multiply hidden ones by 0;
//   * what a row sees is arithmetic: only tiles at an edge of it compare entries, with three thresholds of the row's.
// What it takes, beside the other kernel: at grouped_tc_takes.
// Every wait is bounded; a wait that runs out raises the CTA's abort flag and the device error word, and no row of its block is stored.
#include "attn_tcgen05.cuh"
#include "attn_tile.cuh"
#include "dense.cuh"

namespace b200 {

namespace {

constexpr int GA_M = 128, GA_N = 128, GA_THREADS = 512, GA_ERR_WAIT = 4;
constexpr float GA_LAZY = 8.0f;

template <int D>
struct GaCfg {
    static constexpr int CHUNKS = D / 64, TILE = GA_N * D * 2, SLOTS = D == 128 ? 5 : 8, PITCH = D + 4;
    static constexpr int SMEM = GA_M * D * 2 + SLOTS * TILE + 1024;
    static constexpr uint32_t O_COL = 2 * GA_N;
    static constexpr uint32_t BF = (1u << 4) | (1u << 7) | (1u << 10);   // F32 accumulator, BF16 operands
    static constexpr uint32_t IDESC_S = BF | ((uint32_t)(GA_N >> 3) << 17) | ((uint32_t)(GA_M >> 4) << 24);
    static constexpr uint32_t IDESC_O = BF | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((uint32_t)(GA_M >> 4) << 24);
};
struct GaShared {
    uint64_t full[8], empty[8], sfull[2], pready[2], qready, done;
    float ml[2][GA_M][2];
    uint32_t tmem_base;
    int abort_flag;
};

// the entries a block's rows see: positions 0 .. kept - 1, then lo .. (Entries of grouped_attn.cu)
struct GaEntries {
    int kept, lo, total;
    __device__ __forceinline__ int position(int e) const { return e < kept ? e : lo + e - kept; }
};

template <typename Y, int D>
__global__ void __launch_bounds__(GA_THREADS, 1)
grouped_attn_tc_kernel(const __grid_constant__ CUtensorMap cells, const __grid_constant__ CUtensorMap runs, const GroupedArgs a, int group, bool vec_q, int *err, uint32_t wait_limit, int mute) {
    using C = GaCfg<D>;
    extern __shared__ uint8_t ga_raw[];
    __shared__ GaShared sh;
    pdl_trigger();
    const uint32_t q_s = (pa_smem(ga_raw) + 1023u) & ~1023u, kv_s = q_s + GA_M * D * 2;
    uint8_t *const q_g = ga_raw + (q_s - pa_smem(ga_raw));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    volatile int *abort_flag = &sh.abort_flag;
    const int per = GA_M / group, hk = blockIdx.y;   // tokens of a block
    pdl_wait();
    int r0, tokens;
    // later blocks of a prompt see more keys: they go first
    const int32_t *sg = find_tile(a.seg, a.n_seg, a.n, per, (int)(gridDim.x - 1 - blockIdx.x), &r0, &tokens, err);
    if (!sg) return;
    const int64_t row0 = sg[SEG_ROW0] + r0;
    const int pos0 = sg[SEG_POS0] + r0, last = pos0 + tokens - 1;
    if (a.rot_dims > 0 && (pos0 < 0 || last >= a.rope_rows)) {
        if (tid == 0) atomicExch(err, ERR_POS);
        return;
    }
    const int window = a.window > 0 ? a.window : 0x7fffffff, keep = a.window > 0 ? a.keep : 0;
    GaEntries en;
    en.kept = a.window > 0 ? min(a.keep, last + 1) : 0;
    en.lo = a.window > 0 ? max(a.keep, pos0 - a.window + 1) : 0;
    en.total = en.kept + max(0, last + 1 - en.lo);
    const int tiles = (en.total + GA_N - 1) / GA_N;

    if (tid == 0) {
        for (int i = 0; i < 8; i++) {
            pa_init(&sh.full[i], 1);
            pa_init(&sh.empty[i], 1);
        }
        for (int g = 0; g < 2; g++) {
            pa_init(&sh.sfull[g], 1);
            pa_init(&sh.pready[g], 4);
        }
        pa_init(&sh.qready, 8);
        pa_init(&sh.done, 1);
        sh.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pa_smem(&sh.tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pa_fence_before();
    __syncthreads();
    pa_fence_after();
    const uint32_t tmem = sh.tmem_base;

    if (warp < 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == 1) {
            const bool leader = pa_elect();
            int seq = 0;
            const uint64_t q_desc = pa_desc(q_s, 16), k_desc = pa_desc(kv_s, 16), v_desc = pa_desc(kv_s, GA_N * 128);
            auto wait_slot = [&](int q) {
                const bool ok = pa_wait(&sh.full[q % C::SLOTS], (uint32_t)(q / C::SLOTS) & 1u, abort_flag, wait_limit);
                pa_fence_after();
                return ok;
            };
            // scores of the tile in slot `seq`: over the group's former weights, whose product was issued before (products complete in order)
            auto scores = [&](int g) {
                const int s = seq % C::SLOTS;
                if (leader) {
#pragma unroll
                    for (int ks = 0; ks < D / 16; ks++) {
                        const uint32_t off = (uint32_t)((ks >> 2) * GA_M * 128 + (ks & 3) * 32) >> 4;
                        pa_mma_ss(tmem + (uint32_t)(g * GA_N), q_desc + off, k_desc + (uint32_t)(s * (C::TILE >> 4)) + off, C::IDESC_S, ks > 0);
                    }
                    pa_commit(&sh.empty[s]);
                    pa_commit(&sh.sfull[g]);
                }
                seq++;
            };
            bool ok = pa_wait(&sh.qready, 0, abort_flag, wait_limit);
            for (int g = 0; g < 2 && ok && g < tiles; g++) {
                ok = wait_slot(seq);
                if (ok) scores(g);
            }
            for (int v = 0; v < tiles && ok; v++) {
                const int g = v & 1, j = v >> 1, s = seq % C::SLOTS;
                const bool more = v + 2 < tiles;
                ok = wait_slot(seq) && (!more || wait_slot(seq + 1)) && pa_wait(&sh.pready[g], (uint32_t)j & 1u, abort_flag, wait_limit);
                if (!ok) break;
                pa_fence_after();
                if (leader) {
#pragma unroll
                    for (int part = 0; part < 2; part++)   // the weights' high parts, then their low parts
#pragma unroll
                        for (int ks = 0; ks < GA_N / 16; ks++)
                            pa_mma_ts(tmem + C::O_COL + (uint32_t)(g * D), tmem + (uint32_t)(g * GA_N + part * 64 + ks * 8), v_desc + (uint32_t)(s * (C::TILE >> 4) + ks * 128),
                                      C::IDESC_O, j > 0 || ks > 0 || part > 0);
                    pa_commit(&sh.empty[s]);
                }
                seq++;
                if (more) scores(g);
            }
            if (leader) pa_commit(&sh.done);
            // the operands and tensor memory stay until the products are through, whatever the other roles do
            pa_drain(&sh.done, 0, wait_limit);
        } else if (warp == 0) {
            // keys of tile 0, keys of tile 1, then values of tile v and keys of tile v + 2, the order in which the products read them.  A lane brings four
            // entries' rows, whose cells it has looked up: a row that the lists do not have reads as zeros (and is reported)
            int seq = 0;
            struct Rows { int c[4]; bool run; };   // run: the 32 rows of this lane and its neighbours (eight lanes) stand one after the other
            const auto find = [&](int t) {
                Rows r;
                const int kept = sg[SEG_KEPT], key0 = sg[SEG_KEY0];
                const int64_t tab0 = sg[SEG_TAB0];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int e = t * GA_N + 4 * lane + i, p = en.position(e);
                    const int64_t at = tab0 + (p < kept ? p : kept + p - key0);
                    const bool listed = e < en.total && !(p >= kept && p < key0) && at >= 0 && at < a.n_tab;
                    r.c[i] = listed ? a.tab[at] : -1;
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const bool in = r.c[i] >= 0 && r.c[i] < a.n_cells;
                    if (!in) r.c[i] = -1;
                    if (!in && t * GA_N + 4 * lane + i < en.total) atomicExch(err, ERR_CELL);
                }
                const int base = __shfl_sync(0xffffffffu, r.c[0], lane & ~7);
                const bool mine = base >= 0 && r.c[0] == base + 4 * (lane & 7) && r.c[1] == r.c[0] + 1 && r.c[2] == r.c[0] + 2 && r.c[3] == r.c[0] + 3;
                r.run = (__ballot_sync(0xffffffffu, mine) >> (lane & ~7) & 0xffu) == 0xffu;
                return r;
            };
            const auto load = [&](const Rows &rows, int from, bool muted = false) {
                const int s = seq % C::SLOTS;
                if (!pa_wait(&sh.empty[s], ((uint32_t)(seq / C::SLOTS) & 1u) ^ 1u, abort_flag, wait_limit)) return false;
                if (lane == 0) pa_expect(&sh.full[s], C::TILE);
                __syncwarp();
                const uint32_t dst = kv_s + (uint32_t)(s * C::TILE + lane * 512), bar = pa_smem(&sh.full[s]);
#pragma unroll
                for (int c = 0; c < C::CHUNKS; c++) {
                    if (muted) continue;
                    if (!rows.run)
                        asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst + c * (GA_N * 128)),
                                     "l"(&cells), "r"(from + 64 * c), "r"(rows.c[0]), "r"(rows.c[1]), "r"(rows.c[2]), "r"(rows.c[3]), "r"(bar)
                                     : "memory");
                    else if ((lane & 7) == 0)
                        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst + c * (GA_N * 128)), "l"(&runs),
                                     "r"(from + 64 * c), "r"(rows.c[0]), "r"(bar)
                                     : "memory");
                }
                seq++;
                return true;
            };
            const int keys = hk * 2 * D, values = keys + D;
            Rows r0s = find(0), r1s = find(1);
            bool ok = tiles < 1 || (load(r0s, keys) && (tiles < 2 || load(r1s, keys)));
            for (int v = 0; v < tiles && ok; v++) {
                const Rows next = find(v + 2);   // on their way while a slot is waited for
                ok = load(r0s, values, v == mute && hk == 0 && r0 + tokens == sg[SEG_ROWS]) && (v + 2 >= tiles || load(next, keys));
                r0s = r1s;
                r1s = next;
            }
            // a CTA that gives up still waits (bounded) for the copies it has in flight
            if (*abort_flag)
                for (int q = seq < C::SLOTS ? 0 : seq - C::SLOTS; q < seq; q++) pa_drain(&sh.full[q % C::SLOTS], (uint32_t)(q / C::SLOTS) & 1u, wait_limit);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
        const int g = (warp - 8) >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t t_s = tmem + lanes + (uint32_t)(g * GA_N), t_o = tmem + lanes + C::O_COL + (uint32_t)(g * D);
        {
            // rotated queries as BF16 into the swizzled K-major operand: a warp takes 16 rows, lane = two neighbouring channels of each 64
            const int half = a.rot_dims >> 1;
#pragma unroll 1
            for (int h = 0; h < 16; h += 8) {
                float2 f[8][C::CHUNKS], y[8][C::CHUNKS];
                float4 w[8][C::CHUNKS];   // cos, sin, cos, sin
                // no load behind a branch: rows past the last read the last, channels that are not rotated themselves
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int x = (warp - 8) * 16 + h + u, tok = min(x / group, tokens - 1);
                    const float *q = a.proj + (row0 + tok) * a.ldp + (int64_t)(hk * group + x % group) * D;
                    const float *rope = a.rope + (int64_t)(pos0 + tok) * a.rot_dims;
#pragma unroll
                    for (int c = 0; c < C::CHUNKS; c++) {
                        const int j = 64 * c + 2 * lane, i = j < half ? j : j - half;
                        const bool rot = j < a.rot_dims;
                        const int other = rot ? (j < half ? j + half : j - half) : j;
                        w[u][c] = make_float4(1.0f, 0.0f, 1.0f, 0.0f);
                        if (vec_q) {
                            f[u][c] = *(const float2 *)(q + j);
                            y[u][c] = *(const float2 *)(q + other);
                            if (a.rot_dims > 0) w[u][c] = *(const float4 *)(rope + (rot ? 2 * i : 0));
                        } else {   // of pairs that straddle an edge each channel on its own
                            float v[2];
                            for (int k = 0; k < 2; k++) {
                                const int d = j + k, n = d < half ? d : d - half;
                                v[k] = q[d];
                                if (d < a.rot_dims) v[k] = d < half ? fmaf(v[k], rope[2 * n], -(q[d + half] * rope[2 * n + 1])) : fmaf(v[k], rope[2 * n], q[d - half] * rope[2 * n + 1]);
                            }
                            f[u][c] = make_float2(v[0], v[1]);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int x = (warp - 8) * 16 + h + u;
#pragma unroll
                    for (int c = 0; c < C::CHUNKS; c++) {
                        const int j = 64 * c + 2 * lane;
                        float2 v = f[u][c];
                        if (vec_q && j < a.rot_dims) {
                            const float s1 = j < half ? -1.0f : 1.0f;
                            v = make_float2(fmaf(v.x, w[u][c].x, s1 * (y[u][c].x * w[u][c].y)), fmaf(v.y, w[u][c].z, s1 * (y[u][c].y * w[u][c].w)));
                        }
                        if (x / group >= tokens) v = make_float2(0.0f, 0.0f);
                        *(uint32_t *)(q_g + c * (GA_M * 128) + (x >> 3) * 1024 + (x & 7) * 128 + ((((lane >> 2) ^ (x & 7)) << 4) | (lane & 3) * 4)) = bf16_pack(v.x, v.y);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) pa_arrive(&sh.qready);
        }
        // the entries a row sees: 0 .. h0, and l1 .. h1
        const int p = pos0 + (r / group < tokens ? r / group : 0);
        const int h0 = min(en.kept - 1, p), l1 = max(en.kept, p - window - en.lo + en.kept + 1), h1 = min(en.total - 1, p - en.lo + en.kept);
        const float sc = a.scale * 1.4426950408889634f;   // powers of two
        float m = -INFINITY, l = 0.0f;
        for (int j = 0; 2 * j + g < tiles; j++) {
            const int k0 = (2 * j + g) * GA_N;
            if (!pa_wait(&sh.sfull[g], (uint32_t)j & 1u, abort_flag, wait_limit)) break;
            pa_fence_after();
            uint32_t s[GA_N];
#pragma unroll
            for (int c = 0; c < GA_N; c += 32) pa_ld32(s + c, t_s + (uint32_t)c);
            pa_wait_ld();
            // only tiles at an edge of what the block's rows see need the comparison
            const int pfirst = en.position(k0), plast = en.position(k0 + GA_N - 1);
            const bool edge = k0 + GA_N > en.total || plast > pos0 || (plast >= keep && last - pfirst >= window);
            if (edge) {
#pragma unroll
                for (int c = 0; c < GA_N; c++) {
                    const int e = k0 + c;
                    if (!(e <= h0 || (e >= l1 && e <= h1))) s[c] = 0xff800000u;
                }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < GA_N; c += 8)
#pragma unroll
                for (int e = 0; e < 4; e++) mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(s[c + e]), __uint_as_float(s[c + 4 + e])));
            const float top = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc);
            if (j == 0) {
                m = top;
            } else {
                const bool grow = top > m + GA_LAZY;   // also when nothing was seen before
                if (__any_sync(0xffffffffu, grow)) {
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
            uint64_t ps = 0;
            const uint64_t sc2 = pa_pair(sc, sc), sub2 = pa_pair(-sub, -sub);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t hi[32], lo[32];
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    const float2 x = pa_split(pa_fma2(pa_pair(__uint_as_float(s[64 * h + 2 * c]), __uint_as_float(s[64 * h + 2 * c + 1])), sc2, sub2));
                    const float u = pa_ex2(x.x), v = pa_ex2(x.y);
                    ps = pa_add2(ps, pa_pair(u, v));
                    hi[c] = bf16_pack(u, v);
                    lo[c] = bf16_pack(u - bf16_lo(hi[c]), v - bf16_hi(hi[c]));
                }
                pa_st32(t_s + (uint32_t)(32 * h), hi);
                pa_st32(t_s + (uint32_t)(64 + 32 * h), lo);
            }
            const float2 p2 = pa_split(ps);
            l += p2.x + p2.y;
            pa_wait_st();
            pa_fence_before();
            __syncwarp();
            if (lane == 0) pa_arrive(&sh.pready[g]);
        }
        sh.ml[g][r][0] = m;
        sh.ml[g][r][1] = l;
        const bool finished = __all_sync(0xffffffffu, pa_wait(&sh.done, 0, abort_flag, wait_limit) && !*abort_flag);
        pa_fence_after();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const float ma = sh.ml[0][r][0], mb = sh.ml[1][r][0], mm = fmaxf(ma, mb);
        // no output where the group had no tile or the row saw nothing in them.  Their sum is 0 then, or NaN: a maximum does not show a NaN
        const bool ina = ma != -INFINITY, inb = mb != -INFINITY;
        const float wa = ina ? pa_ex2(ma - mm) : 1.0f, wb = inb ? pa_ex2(mb - mm) : 1.0f;
        const float lt = wa * sh.ml[0][r][1] + wb * sh.ml[1][r][1];
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (g == 0) {
            sh.ml[0][r][0] = mm;
            sh.ml[0][r][1] = lt;
        }
        if (finished) {
            float *part = (float *)(q_g + GA_M * D * 2) + (size_t)r * C::PITCH;   // over the key / value slots
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
    if (*abort_flag) {
        if (tid == 0) atomicExch(err, GA_ERR_WAIT);
        return;
    }
    float sinks[GA_M / 16];   // of the rows warp, warp + 16, ..: all on their way at once
#pragma unroll
    for (int i = 0; i < GA_M / 16; i++) sinks[i] = a.sink ? a.sink[hk * group + (warp + 16 * i) % group] * 1.4426950408889634f : -INFINITY;
    uint32_t again = 0;   // which of this warp's rows are not finite
#pragma unroll
    for (int i = 0; i < GA_M / 16; i++) {
        const int x = warp + 16 * i, tok = x / group, head = hk * group + x - tok * group;
        if (tok >= tokens) break;
        const float m = sh.ml[0][x][0], lt = sh.ml[0][x][1];
        const float mf = fmaxf(m, sinks[i]), w = pa_ex2(m - mf), f = w / (lt * w + pa_ex2(sinks[i] - mf));
        const float *part = (const float *)(q_g + GA_M * D * 2) + (size_t)x * C::PITCH;
        Y *y = (Y *)a.y + (row0 + tok) * a.ldy + (int64_t)head * D;
        bool fine = pa_finite(lt);
#pragma unroll
        for (int c = 0; c < C::CHUNKS; c++) {
            const int j = 64 * c + 2 * lane;
            const float2 v = *(const float2 *)(part + j);
            fine = fine && pa_finite(v.x) && pa_finite(v.y);
            y[j] = from_f32<Y>(v.x * f);
            y[j + 1] = from_f32<Y>(v.y * f);
        }
        if (!__all_sync(0xffffffffu, fine)) again |= 1u << i;
    }
#pragma unroll 1
    for (; again; again &= again - 1) {
        const int x = warp + 16 * (__ffs(again) - 1), tok = x / group, head = hk * group + x - tok * group, p = pos0 + tok;
        const int h0 = min(en.kept - 1, p), l1 = max(en.kept, p - window - en.lo + en.kept + 1), h1 = min(en.total - 1, p - en.lo + en.kept);
        const __nv_bfloat16 *const cache = (const __nv_bfloat16 *)a.cache + (int64_t)hk * 2 * D;
        const int kept = sg[SEG_KEPT], key0 = sg[SEG_KEY0];
        const int64_t tab0 = sg[SEG_TAB0];
        float acc[D / 32], m, lt;
        pa_row_again<D, true>(q_g, x, a.scale * 1.4426950408889634f, en.total, [&](int e, float *, const uint8_t **key, const uint8_t **value) {
            if (!(e <= h0 || (e >= l1 && e <= h1))) return false;
            const int at_pos = en.position(e);
            const int64_t at = tab0 + (at_pos < kept ? at_pos : kept + at_pos - key0);
            if ((at_pos >= kept && at_pos < key0) || at < 0 || at >= a.n_tab || a.tab[at] < 0 || a.tab[at] >= a.n_cells) return false;   // reported above
            *key = (const uint8_t *)(cache + (int64_t)a.tab[at] * a.ldc);
            *value = *key + 2 * D;
            return true;
        }, acc, &m, &lt);
        const float sink = a.sink ? a.sink[head] * 1.4426950408889634f : -INFINITY;
        const float mf = fmaxf(m, sink), w = pa_ex2(m - mf), f = w / (lt * w + pa_ex2(sink - mf));
        Y *y = (Y *)a.y + (row0 + tok) * a.ldy + (int64_t)head * D;
#pragma unroll
        for (int c = 0; c < C::CHUNKS; c++) {
            y[64 * c + 2 * lane] = from_f32<Y>(acc[2 * c] * f);
            y[64 * c + 2 * lane + 1] = from_f32<Y>(acc[2 * c + 1] * f);
        }
    }
}

template <typename Y, int D>
int launch(const GroupedArgs &a, int *err, cudaStream_t s) {
    static bool attr_done[64] = {};
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    B200_REQUIRE(dev >= 0 && dev < 64, "grouped attention: device index %d out of range", dev);
    if (!attr_done[dev]) {
        B200_CUDA(cudaFuncSetAttribute(grouped_attn_tc_kernel<Y, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, GaCfg<D>::SMEM));
        attr_done[dev] = true;
    }
    const int group = a.heads / a.kv_heads, per = GA_M / group;
    const bool vec_q = a.ldp % 2 == 0 && a.rot_dims % 4 == 0 && (((uintptr_t)a.proj | (uintptr_t)a.rope) & 15) == 0;
    CUtensorMap cells, runs;
    int rc = rows_map(&runs, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.cache, a.ldc, a.n_cells, a.ldc, 32);
    if (rc != B200_STATUS_SUCCESS) return rc;
    rc = rows_map(&cells, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.cache, a.ldc, a.n_cells, a.ldc, 1);   // one row high: rows are gathered
    if (rc != B200_STATUS_SUCCESS) return rc;
    uint32_t wait_limit;
    int mute;
    attn_wait_hook(&wait_limit, &mute);
    return launch_pdl(grouped_attn_tc_kernel<Y, D>, dim3((unsigned)((a.n + per - 1) / per + a.n_seg), (unsigned)a.kv_heads), dim3(GA_THREADS), GaCfg<D>::SMEM, s, cells, runs, a, group, vec_q,
                      err, wait_limit, mute);
}

}  // namespace

// Which prompts: from 256 rows that fill the blocks of their sequences.  A launch costs about 25 us before its second wave of tiles (its code comes into
// the SMs, q is rotated, the first cells are looked up), a tile then 1.5, where the mma.sync kernel's 64 x 64 tiles take long but start at once.
// Whole prompts of 4 layers, us, that kernel / this one: 4096 wide (8 key heads of 128, 32 query heads) 128 rows 990 / 1049, 256 1078 / 1065, 512
// 1272 / 1205, 2048 3535 / 3201; 1024 wide 256 rows 483 / 457, 1100 807 / 626, 2048 962 / 724.
bool grouped_tc_takes(const GroupedArgs &a) {
    const int group = a.heads / a.kv_heads;
    return a.dim == a.vdim && (a.dim == 64 || a.dim == 128) && group <= GA_M && (group & (group - 1)) == 0 && a.n >= 256 && a.n >= 64 * a.n_seg && a.n_cells <= 0x7fffffffLL &&
           a.ldc <= 0x7fffffffLL && a.scale >= 0.0f;
}
int launch_grouped_attn_tc(const GroupedArgs &a, int *err, cudaStream_t s) {
    if (a.dim == 64) return a.y_type == B200_TYPE_F32 ? launch<float, 64>(a, err, s) : launch<__nv_bfloat16, 64>(a, err, s);
    return a.y_type == B200_TYPE_F32 ? launch<float, 128>(a, err, s) : launch<__nv_bfloat16, 128>(a, err, s);
}

}  // namespace b200
